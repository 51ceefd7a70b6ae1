// spiffe_b200/csrc/multigrid_f32.cu -- multigrid Poisson solve of the split-precision form.
//
// The problem is solve_poisson_cyl's (poisson.c:17-130): the five-point
// cylindrical operator on the nodes that routine updates (rows lo..hi,
// columns 0..nr-2, not metal; the axis row of coefficients 4c and e - 2c;
// mirrored end rows for a "Dirichlet" end), every other node held.  The
// reference relaxes it with red-black SOR to its stop rule
// sum|residual| < accuracy sum|rhs|; on the meshes of the RF and DC guns
// that rule is out of reach within its 1000 half-sweeps.  Here the same
// equations are solved by FP64 iterative refinement around FP32 multigrid
// V-cycles:
//
//   r = rhs - A Psi in FP64; stop when sum|r| < accuracy * sum|rhs|
//   (sum|rhs| over iz < nz, ir < nr-1, as poisson.c:40-43 forms it; a
//   Laplace solve, rhs absent, measures against its first residual);
//   u = V-cycle(r) in FP32;  Psi += u in FP64;  repeat.
//
// Levels: level 0 is the mesh; level l+1 holds the nodes 2I, 2J of level l
// (node (I, J) of level l+1 is unknown when node (2I, 2J) of level l is).
// Transfers are bilinear interpolation P and its volume-weighted adjoint
// R = (1/4) Vc^-1 P^T Vf (Vf, Vc: annulus volumes, the axis node's 1/8 of
// the first ring's), and the coarse operators are the Galerkin products
// R A P, built once per mesh on the host in FP64 (nine-point stencils).
// Metal irises and electrodes stay in the coarse operators that way;
// operators rediscretised on the coarse nodes instead lose them and the
// V-cycle then reduces the residual only 0.6x per cycle on the 1.6-cell gun
// against 0.1-0.17x with the Galerkin operators.  Smoothing is red-black
// Gauss-Seidel on level 0 and four-colour Gauss-Seidel (colour (I&1, J&1))
// on the nine-point levels, nu sweeps before and after each coarse
// correction; the last pre-smoothing colour leaves a zero residual at its
// own nodes, so the restriction evaluates the residual only at the others.
//
// A solve is one CUDA graph: a kernel for level 0's residual and way down,
// then a WHILE node around a V-cycle of one kernel a level and direction that
// ends with the next residual; the last CTA of that kernel adds the sums in a
// fixed order and decides whether the loop goes on, so the decision does not
// depend on timing and the host is not asked.  What bounded the previous
// form (one cooperative launch with a grid barrier between colour sweeps,
// about 51 a V-cycle) was those barriers with the L2 round trips between
// them, 3.5 to 7 us each; DRAM was 1 % busy.  Here a kernel works a band of
// rows of its level in shared memory through all sweeps of its direction: it
// loads the band and a halo of one row per row the sweeps reach (five on the
// way down, from u = 0; four up), recomputes the neighbours' values in the
// halo instead of fetching them, and so needs no exchange until the next
// kernel.  Separate kernels rather than phases of one, because each then has
// the registers it needs (in one kernel the compiler spilled, and with most
// of the SM's memory taken as shared memory the spills went to L2: the same
// phases took two to three times as long) and because no CTA waits for
// another, so solves of several instances share the SMs.  Values and update
// order are those of the sweeps run over the whole mesh.
// The first level of at most MG_MAX_DIRECT unknowns is the coarsest, solved
// exactly by its precomputed inverse over the whole GPU.  Coefficients are kept
// per distinct row (class): in a gun nearly all rows of a level are alike, so
// a band's fit L1 and a thread keeps its columns' in registers.
// Within a cycle a kernel comes onto the SMs while the one before ends
// (programmatic edges, step_begin) and has its coefficients in registers by
// the time that has ended (5 to 9 % of a cycle).
// Measured from a cold start to 1e-6 (B200), first form -> here: 3001 x 821
// gun 1.6 -> 0.75 ms in 5 cycles, 1500 x 400 1.13 -> 0.35 in 5, 424 x 232
// 0.99 -> 0.46 in 9, 601 x 165 0.69 -> 0.27 in 5.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <system_error>
#include <thread>
#include <unordered_map>
#include <vector>

#include "modules.cuh"
#include "split32.cuh"

namespace {

constexpr int MG_NT = 512;             // threads per CTA
constexpr int MG_W = MG_NT / 32;       // warps per CTA
constexpr int MG_MIN_UNKNOWNS = 64;    // a mesh of no more unknowns is not coarsened
constexpr int MG_NODES_PER_CTA = 4096; // mesh nodes per band below one band per SM
constexpr int MG_MIN_ROWS = 4;         // own rows of a coarse level's band at least
constexpr int MG_MAX_DIRECT = 2048;    // a level of at most this many unknowns is the coarsest, solved exactly
constexpr int MG_MAX_BAND = 512;       // where the unknowns' couplings reach no farther than this
constexpr int MG_COARSE_SWEEPS = 24;   // sweeps on another coarsest level
constexpr int MG_DOWN = 5, MG_UP = 4;  // halo rows a side of a band on the way down and up
enum { MG_INVD = 8, MG_DIAG = 9 };

// One solve's arguments and its state between the graph's kernels.
struct MgCall {
  double *Psi;
  const double *rhs; // null: Laplace solve
  const uint8_t *umask;
  double accuracy, drive;
  long long max_cycles, cycles;
  PcState *st;
  long long *iters_out;
  DevCounts *cnt;
  unsigned ticket; // bands of the residual that are done
  int skip;
};

// Level 0's size, update region and operator.
struct Mg0 {
  int nz, P, lo, hi, cols;
  int rp, nb;                     // rows of a band, bands
  float a, e, e2c, inv_e, inv_e2c;
  double a_d, e_d, e2c_d;         // in FP64 for the residual
  float *u, *f;                   // the pre-smoothed u and f (NaN where no equation holds) of every row
  const float *crow, *drow;       // the radial couplings of a column in FP32, P values
  const double *cpd, *cmd;        // and in FP64
  double *part;                   // the bands' sums, two a band
};

__device__ __forceinline__ float4 ldcg4(const float *p) { return __ldcg(reinterpret_cast<const float4 *>(p)); }
__device__ __forceinline__ void st4(float *p, float4 v) { *reinterpret_cast<float4 *>(p) = v; }
__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }

extern __shared__ float4 mg_smem[];

// A CTA's buffer: its shared memory, or its part of `scratch` for meshes whose bands do not fit there.
template <bool SM> __device__ __forceinline__ float *band_buf(float *scratch, size_t scratch_n)
{
  return SM ? reinterpret_cast<float *>(mg_smem) : scratch + (size_t)blockIdx.x * scratch_n;
}

// ---- level 0: the mesh, five-point operator.  A band buffer holds rows r0,
// r0+1, ... of u (U) and f (F) at the mesh pitch P0, each row as its even
// columns and then (from H = P0/2) its odd ones, so that the nodes of one
// colour in a row are consecutive; u0 and f0 have the same layout.  f is NaN
// at a node without an equation (metal, outside rows lo..hi, columns >= cols),
// whose u stays 0.

// A thread's share of level 0: four consecutive nodes of a half row (eight
// columns) in rows g, g+groups, ..., their radial couplings in registers.
struct Part0 {
  int j, g, groups; // first half-column; row group; j < 0: no share
  float cE[4], dE[4], cO[4], dO[4]; // couplings outwards and inwards, even and odd columns
  float inv0, e0;                   // 1/e and e of the first even column (the axis has its own)
};

// column groups of level 0
__device__ __forceinline__ int cols0(const Mg0 &z) { return (((z.cols + 1) >> 1) + 3) >> 2; }

__device__ __forceinline__ void part0(const Mg0 &z, Part0 &t, int kb)
{
  const int n = cols0(z), W = (n + 31) & ~31; // padded to whole warps
  t.groups = W < MG_NT ? MG_NT / W : 1;
  t.g = W < MG_NT ? threadIdx.x / W : 0;
  const int k = kb + (int)threadIdx.x - t.g * W;
  t.j = k < n && t.g < t.groups ? 4 * k : -1;
  if (t.j < 0)
    return;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    t.cE[q] = __ldg(z.crow + 2 * (t.j + q));
    t.dE[q] = __ldg(z.drow + 2 * (t.j + q));
    t.cO[q] = __ldg(z.crow + 2 * (t.j + q) + 1);
    t.dO[q] = __ldg(z.drow + 2 * (t.j + q) + 1);
  }
  t.inv0 = t.j ? z.inv_e : z.inv_e2c;
  t.e0 = t.j ? z.e : z.e2c;
}

template <bool RES>
__device__ __forceinline__ void strip0(const Mg0 &z, const Part0 &t, float *U, float *F, int r0, int sa, int sb,
                                       int c)
{
  if (t.j < 0)
    return;
  const int P = z.P, H = P >> 1;
  for (int s = sa + t.g; s < sb; s += t.groups) {
    const int iz = r0 + s, h = (iz ^ c) & 1; // the colour's columns have parity h
    float *row = U + s * P;
    float *x = row + h * H + t.j;
    const bool top = iz == z.nz - 1 && z.hi == z.nz - 1, bottom = iz == 0 && z.lo == 0;
    const float4 um = ld4(top ? x - P : x + P), dm = ld4(bottom ? x + P : x - P);
    const float4 o = ld4(row + (1 - h) * H + t.j), f = ld4(F + s * P + h * H + t.j);
    float nb[4];
    if (h) {
      const float right = row[t.j + 4];
      nb[0] = z.a * (um.x + dm.x) + t.cO[0] * o.y + t.dO[0] * o.x;
      nb[1] = z.a * (um.y + dm.y) + t.cO[1] * o.z + t.dO[1] * o.y;
      nb[2] = z.a * (um.z + dm.z) + t.cO[2] * o.w + t.dO[2] * o.z;
      nb[3] = z.a * (um.w + dm.w) + t.cO[3] * right + t.dO[3] * o.w;
    } else {
      const float left = t.j ? row[H + t.j - 1] : 0.f;
      nb[0] = z.a * (um.x + dm.x) + t.cE[0] * o.x + t.dE[0] * left;
      nb[1] = z.a * (um.y + dm.y) + t.cE[1] * o.y + t.dE[1] * o.x;
      nb[2] = z.a * (um.z + dm.z) + t.cE[2] * o.z + t.dE[2] * o.y;
      nb[3] = z.a * (um.w + dm.w) + t.cE[3] * o.w + t.dE[3] * o.z;
    }
    float4 v;
    if (RES) {
      const float4 u = ld4(x);
      v.x = f.x - nb[0] - (h ? z.e : t.e0) * u.x;
      v.y = f.y - nb[1] - z.e * u.y;
      v.z = f.z - nb[2] - z.e * u.z;
      v.w = f.w - nb[3] - z.e * u.w;
    } else {
      v.x = (f.x - nb[0]) * (h ? z.inv_e : t.inv0);
      v.y = (f.y - nb[1]) * z.inv_e;
      v.z = (f.z - nb[2]) * z.inv_e;
      v.w = (f.w - nb[3]) * z.inv_e;
    }
    v.x = f.x == f.x ? v.x : 0.f;
    v.y = f.y == f.y ? v.y : 0.f;
    v.z = f.z == f.z ? v.z : 0.f;
    v.w = f.w == f.w ? v.w : 0.f;
    st4(RES ? F + s * P + h * H + t.j : x, v);
  }
}

// One colour c ((iz+ir)%2 == c) of red-black Gauss-Seidel on rows r0+sa ..
// r0+sb-1; with RES the residual f - A u of that colour into F instead (0
// without an equation).  A mesh wider than the CTA takes its columns in strips.
template <bool RES>
__device__ __forceinline__ void relax0(const Mg0 &z, Part0 &t, float *U, float *F, int r0, int sa, int sb, int c)
{
  const int n = cols0(z);
  for (int kb = 0;;) {
    strip0<RES>(z, t, U, F, r0, sa, sb, c);
    if ((kb += MG_NT) >= n)
      break;
    part0(z, t, kb);
  }
  if (n > MG_NT)
    part0(z, t, 0);
}

// ---- levels >= 1: nine-point Galerkin operators.  A row holds its even
// columns, then (from Q) its odd ones, each half with a halo column: node J
// at (J&1) Q + (J>>1) + 1.
__device__ __forceinline__ int col9(const MgLevel &L, int J) { return (J & 1) * L.Q + (J >> 1) + 1; }

// The coefficients of the node pair (2j, 2j+1) of a row of class v.
struct Coef9 {
  float c0[8], c1[8];
};

__device__ __forceinline__ const float *load_coef9(const MgLevel &L, int v, int j, Coef9 &c)
{
  int P = L.P; // opaque here: else the offsets are kept in registers all along
  asm volatile("" : "+r"(P));
  const float *p = L.coef + (size_t)v * (MG_NCOEF * P) + 1 + j;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    c.c0[k] = __ldg(p + k * P);
    c.c1[k] = __ldg(p + k * P + (P >> 1));
  }
  return p;
}

// The neighbours' terms at the pair's node of parity CR (0 even, 1 odd); u: its row
template <int CR> __device__ __forceinline__ float nb9(const MgLevel &L, int j, const Coef9 &k, const float *u)
{
  const int P = L.P, at = (CR ? L.Q + 1 : 1) + j, lf = (CR ? 1 : L.Q) + j;
  const float *c = CR ? k.c1 : k.c0;
  float s = c[0] * u[lf - P];
  s += c[1] * u[at - P];
  s += c[2] * u[lf + 1 - P];
  s += c[3] * u[lf];
  s += c[4] * u[lf + 1];
  s += c[5] * u[lf + P];
  s += c[6] * u[at + P];
  s += c[7] * u[lf + 1 + P];
  return s;
}

// The bilinear correction from level C (row -1 at w) at the pair (i, 2j),
// (i, 2j+1) of the level above (linear along a direction C does not coarsen:
// the node itself).
template <bool CG>
__device__ __forceinline__ void interp(const MgLevel &C, const float *w, int i, int j, float &even, float &odd)
{
  auto at = [&](const float *p) { return CG ? __ldcg(p) : *p; };
  const bool hz = C.cz == 2 && (i & 1); // a half-way row
  const float *p = w + (size_t)((C.cz == 2 ? i >> 1 : i) + 1) * C.P;
  const int k0 = C.cr == 2 ? col9(C, j) : 1 + j, k1 = C.cr == 2 ? col9(C, j + 1) : C.Q + 1 + j;
  const float x = at(p + k0), y = at(p + k1);
  even = x;
  odd = C.cr == 2 ? 0.5f * (x + y) : y;
  if (hz) {
    const float x2 = at(p + C.P + k0), y2 = at(p + C.P + k1);
    even = 0.5f * even + 0.5f * x2;
    odd = 0.5f * odd + 0.5f * (C.cr == 2 ? 0.5f * (x2 + y2) : y2);
  }
}

// A thread's share of the rows rlo <= I < rhi of a nine-point level in a
// buffer whose first row is r0.  The coefficients of a held node are all 0,
// so its u comes out 0.
//
// Fix9: up to K node pairs of the even rows and K of the odd ones, with their
// coefficients and f/diagonal in registers for the whole visit.  For the
// levels and bands with at most K MG_NT pairs of a row parity, where a colour
// step is a chain of latencies: shared-memory loads, eight fused
// multiply-adds, a barrier.
template <int K> struct Fix9 {
  int at[2][K], row[2][K], j[2][K]; // place of the row; row (INT_MIN: none)
  Coef9 c[2][K];
  float g0[2][K], g1[2][K]; // f/diagonal
  unsigned unk;             // bits 2 (K parity + k), +1: the pair's even and odd nodes are unknowns

  // init: what is constant (before the kernel's turn has come); start: f
  __device__ __forceinline__ void init(const MgLevel &L, int r0, int rlo, int rhi)
  {
    const int n = (L.R + 1) >> 1;
    rlo = max(rlo, 0);
    rhi = min(rhi, L.Z);
    unk = 0;
#pragma unroll
    for (int z = 0; z < 2; z++)
#pragma unroll
      for (int k = 0; k < K; k++) {
        const int t = threadIdx.x + k * MG_NT, q = (unsigned)t / (unsigned)n, I = rlo + ((rlo ^ z) & 1) + 2 * q;
        row[z][k] = INT_MIN;
        if (I < rhi) {
          row[z][k] = I;
          j[z][k] = t - q * n;
          at[z][k] = (I - r0) * L.P;
          const float *p = load_coef9(L, __ldg(L.cls + I), j[z][k], c[z][k]);
          const float i0 = g0[z][k] = __ldg(p + MG_INVD * L.P), i1 = g1[z][k] = __ldg(p + MG_INVD * L.P + L.Q);
          unk |= (i0 != 0.f ? 1u : 0u) << (2 * (K * z + k)) | (i1 != 0.f ? 2u : 0u) << (2 * (K * z + k));
        }
      }
  }
  __device__ __forceinline__ void start(const MgLevel &L, const float *F)
  {
#pragma unroll
    for (int z = 0; z < 2; z++)
#pragma unroll
      for (int k = 0; k < K; k++)
        if (row[z][k] != INT_MIN) {
          g0[z][k] *= F[at[z][k] + 1 + j[z][k]];
          g1[z][k] *= F[at[z][k] + L.Q + 1 + j[z][k]];
        }
  }
  template <int CZ, int CR>
  __device__ __forceinline__ void colour(const MgLevel &L, float *U, const float *, int, int ra, int rb)
  {
#pragma unroll
    for (int k = 0; k < K; k++)
      if (row[CZ][k] >= ra && row[CZ][k] < rb) {
        float *u = U + at[CZ][k];
        u[(CR ? L.Q + 1 : 1) + j[CZ][k]] = (CR ? g1[CZ][k] : g0[CZ][k]) - nb9<CR>(L, j[CZ][k], c[CZ][k], u);
      }
  }
  __device__ __forceinline__ void resid(const MgLevel &L, const float *U, const float *, float *R, int, int ra, int rb)
  {
#pragma unroll
    for (int z = 0; z < 2; z++)
#pragma unroll
      for (int k = 0; k < K; k++)
        if (row[z][k] >= ra && row[z][k] < rb) {
          const float *u = U + at[z][k];
          const float *d = L.coef + (size_t)(__ldg(L.cls + row[z][k]) * MG_NCOEF + MG_DIAG) * L.P;
          const int a0 = 1 + j[z][k], a1 = L.Q + 1 + j[z][k];
          const float e = __ldg(d + a0) * (g0[z][k] - nb9<0>(L, j[z][k], c[z][k], u) - u[a0]);
          const float o = __ldg(d + a1) * (g1[z][k] - nb9<1>(L, j[z][k], c[z][k], u) - u[a1]);
          R[at[z][k] + a0] = e;
          R[at[z][k] + a1] = o;
        }
  }
  template <bool CG>
  __device__ __forceinline__ void prolong(const MgLevel &L, const MgLevel &C, float *U, const float *w, int)
  {
#pragma unroll
    for (int z = 0; z < 2; z++)
#pragma unroll
      for (int k = 0; k < K; k++)
        if (row[z][k] != INT_MIN) {
          float e, o;
          interp<CG>(C, w, row[z][k], j[z][k], e, o);
          float *u = U + at[z][k] + 1 + j[z][k];
          if (unk >> (2 * (K * z + k)) & 1)
            u[0] += e;
          if (unk >> (2 * (K * z + k)) & 2)
            u[L.Q] += o;
        }
  }
};

// Run9: one pair of columns in a run of rows, MG_ROWS of a parity at a time
// (their loads overlap); the coefficients of a class in registers, loaded
// again where a run's classes differ (at metal edges).  A level wider than
// the CTA takes its columns in strips.
constexpr int MG_ROWS = 3;
struct Run9 {
  int j, lo, hi, W, n, v; // columns 2j, 2j+1 (j < 0: none); rows; lanes a row group; pairs a row; class
  Coef9 c;
  float i0, i1;

  __device__ __forceinline__ void strip(int jb)
  {
    const int k = W < MG_NT ? (int)threadIdx.x % W : jb + (int)threadIdx.x;
    j = k < n ? k : -1;
    v = -1;
  }
  __device__ __forceinline__ void start(const MgLevel &, const float *) {}
  __device__ __forceinline__ void init(const MgLevel &L, int, int rlo, int rhi)
  {
    n = (L.R + 1) >> 1;
    W = (n + 31) & ~31;
    rlo = max(rlo, 0);
    rhi = min(rhi, L.Z);
    const int groups = W < MG_NT ? MG_NT / W : 1, g = W < MG_NT ? (int)threadIdx.x / W : 0;
    const int per = (rhi - rlo + groups - 1) / groups;
    lo = rlo + g * per;
    hi = g < groups ? min(lo + per, rhi) : lo;
    strip(0);
  }
  __device__ __forceinline__ void load(const MgLevel &L, int cls)
  {
    if (cls == v)
      return;
    v = cls;
    const float *p = load_coef9(L, cls, j, c);
    i0 = __ldg(p + MG_INVD * L.P);
    i1 = __ldg(p + MG_INVD * L.P + L.Q);
  }
  template <class Fn> __device__ __forceinline__ void strips(Fn fn)
  {
    for (int jb = 0;;) {
      if (j >= 0)
        fn();
      if ((jb += MG_NT) >= n)
        break;
      strip(jb);
    }
    if (n > MG_NT)
      strip(0);
  }
  template <int CZ, int CR>
  __device__ __forceinline__ void colour(const MgLevel &L, float *U, const float *F, int r0, int ra, int rb)
  {
    strips([&]() {
      const int a = max(lo, ra), b = min(hi, rb), at = (CR ? L.Q + 1 : 1) + j;
#pragma unroll 1
      for (int I = a + ((a ^ CZ) & 1); I < b; I += 2 * MG_ROWS) {
        int cl[MG_ROWS];
#pragma unroll
        for (int k = 0; k < MG_ROWS; k++)
          cl[k] = __ldg(L.cls + min(I + 2 * k, b - 1));
        bool same = true;
#pragma unroll
        for (int k = 1; k < MG_ROWS; k++)
          same = same && (I + 2 * k >= b || cl[k] == cl[0]);
        float *u = U + (I - r0) * L.P;
        const float *f = F + (I - r0) * L.P + at;
        if (same && I + 2 * (MG_ROWS - 1) < b) {
          load(L, cl[0]);
          float x[MG_ROWS];
#pragma unroll
          for (int k = 0; k < MG_ROWS; k++)
            x[k] = f[2 * k * L.P] * (CR ? i1 : i0) - nb9<CR>(L, j, c, u + 2 * k * L.P);
#pragma unroll
          for (int k = 0; k < MG_ROWS; k++)
            u[2 * k * L.P + at] = x[k];
        } else {
#pragma unroll 1
          for (int k = 0; k < MG_ROWS && I + 2 * k < b; k++) {
            load(L, __ldg(L.cls + I + 2 * k));
            u[2 * k * L.P + at] = f[2 * k * L.P] * (CR ? i1 : i0) - nb9<CR>(L, j, c, u + 2 * k * L.P);
          }
        }
      }
    });
  }
  __device__ __forceinline__ void resid(const MgLevel &L, const float *U, const float *F, float *R, int r0, int ra,
                                        int rb)
  {
    strips([&]() {
      const int a0 = 1 + j, a1 = L.Q + 1 + j;
#pragma unroll 1
      for (int I = max(lo, ra); I < min(hi, rb); I++) {
        load(L, __ldg(L.cls + I));
        const float *u = U + (I - r0) * L.P, *f = F + (I - r0) * L.P;
        const float *d = L.coef + (size_t)(v * MG_NCOEF + MG_DIAG) * L.P;
        const float e = __ldg(d + a0) * (f[a0] * i0 - nb9<0>(L, j, c, u) - u[a0]);
        const float o = __ldg(d + a1) * (f[a1] * i1 - nb9<1>(L, j, c, u) - u[a1]);
        R[(I - r0) * L.P + a0] = e;
        R[(I - r0) * L.P + a1] = o;
      }
    });
  }
  template <bool CG>
  __device__ __forceinline__ void prolong(const MgLevel &L, const MgLevel &C, float *U, const float *w, int r0)
  {
    strips([&]() {
#pragma unroll 1
      for (int I = lo; I < hi; I += 4) {
        float e[4], o[4];
        int cl[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
          cl[k] = __ldg(L.cls + min(I + k, hi - 1));
          interp<CG>(C, w, min(I + k, hi - 1), j, e[k], o[k]);
        }
#pragma unroll
        for (int k = 0; k < 4; k++)
          if (I + k < hi) {
            load(L, cl[k]);
            float *u = U + (I + k - r0) * L.P + 1 + j;
            if (i0 != 0.f)
              u[0] += e[k];
            if (i1 != 0.f)
              u[L.Q] += o[k];
          }
      }
    });
  }
};

// Both colours of row parity CZ on rows ra <= I < rb, column parity CR
// first: the second reads the first only in its own row, so a CTA barrier
// lies between them.
template <int CZ, int CR, class Op>
__device__ __forceinline__ void rows9(const MgLevel &L, Op &t, float *U, const float *F, int r0, int ra, int rb)
{
  t.template colour<CZ, CR>(L, U, F, r0, ra, rb);
  __syncthreads();
  t.template colour<CZ, 1 - CR>(L, U, F, r0, ra, rb);
  __syncthreads();
}

// f of level C's rows Ia .. Ib-1 from the residual R (a buffer whose first
// row is r0) of the level L above, into rows of pitch C.P from `out` on (row
// -1 first); a thread keeps a column.  Halo rows and columns of R are 0.
__device__ __forceinline__ void restrict9(const MgLevel &L, const MgLevel &C, const float *R, int r0, int Ia, int Ib,
                                          float *out)
{
  const int W = (C.R + 31) & ~31, groups = W < MG_NT ? MG_NT / W : 1, g = W < MG_NT ? threadIdx.x / W : 0, P = L.P;
  if (g >= groups)
    return;
  for (int J = threadIdx.x - g * W; J < C.R; J += MG_NT) {
    const int k = col9(C, J), j = C.cr * J, at = col9(L, j), l = col9(L, j - 1), r = col9(L, j + 1);
    const float w0 = C.cr == 2 ? __ldg(C.rw + 3 * J) : 0.f, w1 = __ldg(C.rw + 3 * J + 1);
    const float w2 = C.cr == 2 ? __ldg(C.rw + 3 * J + 2) : 0.f, wz = C.cz == 2 ? 0.5f * w1 : 0.f;
#pragma unroll 1
    for (int I = Ia + g; I < Ib; I += groups) {
      const float *x = R + (C.cz * I - r0) * P;
      float v = w1 * x[at];
      if (C.cr == 2)
        v += w0 * x[l] + w2 * x[r];
      if (C.cz == 2)
        v += wz * x[at - P] + wz * x[at + P];
      out[(I + 1) * C.P + k] = v;
    }
  }
}

// The same from level 0's residual in a band buffer.  Level 0's last colour
// (1) has a zero residual, so only its (iz+ir) even nodes count.
__device__ __forceinline__ void restrict0(const MgLevel &C, int P, const float *R, int r0, int Ia, int Ib, float *out)
{
  const int W = (C.R + 31) & ~31, groups = W < MG_NT ? MG_NT / W : 1, g = W < MG_NT ? threadIdx.x / W : 0, H = P >> 1;
  if (g >= groups)
    return;
  for (int J = threadIdx.x - g * W; J < C.R; J += MG_NT) {
    const int k = col9(C, J);
    const float w0 = J ? __ldg(C.rw + 3 * J) : 0.f, w1 = __ldg(C.rw + 3 * J + 1), w2 = __ldg(C.rw + 3 * J + 2);
    const int in = J ? 1 : 0; // the inner neighbour (none on the axis)
#pragma unroll 1
    for (int I = Ia + g; I < Ib; I += groups) {
      const float *x = R + (C.cz * I - r0) * P;
      float v;
      if (C.cz == 2 && C.cr == 2) { // row 2I, column 2J; rows 2I +- 1, columns 2J -+ 1
        const float *y = x + H + J;
        v = w1 * x[J] + 0.5f * w2 * (y[-P] + y[P]) + 0.5f * w0 * (y[-P - in] + y[P - in]);
      } else if (C.cz == 2) { // coarsened in z only: the column has the colour in every other row
        const int at = (J & 1) * H + (J >> 1);
        v = (J & 1) == 0 ? w1 * x[at] : 0.5f * w1 * (x[at - P] + x[at + P]);
      } else { // in r only: column 2J in even rows, 2J -+ 1 in odd ones
        const float *y = x + H + J;
        v = (I & 1) == 0 ? w1 * x[J] : w2 * y[0] + w0 * y[-in];
      }
      // (NaN: R of columns without equations, which only held nodes reach)
      out[(I + 1) * C.P + k] = v == v ? v : 0.f;
    }
  }
}

// ---- the kernels of a V-cycle

__global__ void k_mg_begin(MgCall c, MgCall *call)
{
  c.skip = c.st && !c.st->do_solve;
  *call = c;
}

// CTA sums of two doubles in a fixed order; thread 0 has them
__device__ __forceinline__ double2 block_sums(double x, double y)
{
  __shared__ double sh[2][MG_W];
  for (int o = 16; o > 0; o >>= 1) {
    x += __shfl_down_sync(0xffffffffu, x, o);
    y += __shfl_down_sync(0xffffffffu, y, o);
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) {
    sh[0][w] = x;
    sh[1][w] = y;
  }
  __syncthreads();
  double2 s = make_double2(0, 0);
  if (threadIdx.x == 0)
    for (int k = 0; k < MG_W; k++) {
      s.x += sh[0][k];
      s.y += sh[1][k];
    }
  return s;
}

// Level 0, the residual of the rows a0 .. b0-1 of a band and of MG_DOWN halo
// rows a side (the neighbours' values, formed again here): r = rhs - A Psi in
// FP64, f = r in FP32 and u as the first colour-0 sweep from u = 0 leaves it
// (f/e: the neighbour sum is zero).  Returns this thread's sum |r| and sum
// |rhs| over the own rows (iz < nz, ir < nr-1).  A thread forms the columns
// 2j, 2j+1 and walks down a run of rows, so each Psi is read once, with the
// loads of MG_AHEAD rows in flight together.
constexpr int MG_AHEAD = 4;
__device__ __forceinline__ double2 resid0(const Mg0 &z, const double *Psi, const double *rhs, const uint8_t *umask,
                                          float *U, float *F, int a0, int b0)
{
  const int P = z.P, H = P >> 1, lane = threadIdx.x & 31, r0 = a0 - MG_DOWN, n = b0 - a0 + 2 * MG_DOWN;
  double r_acc = 0, d_acc = 0;
  const float nan = __int_as_float(0x7fc00000);
  const int W = min((H + 31) & ~31, MG_NT), groups = MG_NT / W, g = threadIdx.x / W;
  if (g < groups) {
    const int per = (n + groups - 1) / groups, s0 = g * per, s1 = min(s0 + per, n);
    for (int jl = threadIdx.x - g * W; jl - lane < H; jl += W) {
      const int j = min(jl, H - 1), c0 = 2 * j;
      const double2 cp = __ldg(reinterpret_cast<const double2 *>(z.cpd + c0));
      const double2 cm = __ldg(reinterpret_cast<const double2 *>(z.cmd + c0));
      const double e0 = c0 ? z.e_d : z.e2c_d;
      const bool edge = lane == 0 || lane == 31; // lanes whose outer neighbour column is another warp's
      const int beside = lane ? (c0 + 2 < P ? 2 : 0) : (c0 ? -1 : 0);
      const bool le = c0 < z.cols, lo = c0 + 1 < z.cols;
      auto row = [&](int s) { return min(max(r0 + s, 0), z.nz) * P + c0; }; // fewer than 2^31 nodes
      auto psi = [&](int s) { return __ldcg(reinterpret_cast<const double2 *>(Psi + row(s))); };
      double2 below = psi(s0 - 1), here = psi(s0);
#pragma unroll 1
      for (int sb = s0; sb < s1; sb += MG_AHEAD) {
        double2 nx[MG_AHEAD], rh[MG_AHEAD];
        double sd[MG_AHEAD];
        uchar2 mk[MG_AHEAD];
#pragma unroll
        for (int k = 0; k < MG_AHEAD; k++) {
          const int at = row(sb + k);
          nx[k] = psi(sb + k + 1);
          mk[k] = __ldg(reinterpret_cast<const uchar2 *>(umask + at));
          rh[k] = rhs ? __ldg(reinterpret_cast<const double2 *>(rhs + at)) : make_double2(0, 0);
          sd[k] = edge ? __ldcg(Psi + at + beside) : 0.0;
        }
#pragma unroll
        for (int k = 0; k < MG_AHEAD; k++) {
          const int s = sb + k, iz = r0 + s;
          double left = __shfl_up_sync(0xffffffffu, here.y, 1), right = __shfl_down_sync(0xffffffffu, here.x, 1);
          left = lane == 0 ? sd[k] : left;
          right = lane == 31 ? sd[k] : right;
          const bool own = iz >= a0 && iz < b0 && s < s1, in = iz >= z.lo && iz <= z.hi;
          const double2 up = iz == z.nz - 1 && z.hi == z.nz - 1 ? below : nx[k], dn = iz == 0 && z.lo == 0 ? nx[k] : below;
          const double re = rh[k].x - (z.a_d * (up.x + dn.x) + cp.x * here.y + cm.x * left + e0 * here.x);
          const double ro = rh[k].y - (z.a_d * (up.y + dn.y) + cp.y * right + cm.y * here.x + z.e_d * here.y);
          const bool ve = in && le && !(mk[k].x & S32_U_METAL), vo = in && lo && !(mk[k].y & S32_U_METAL);
          if (jl < H && s < s1) {
            const float fe = ve ? (float)re : nan, fo = vo ? (float)ro : nan;
            if (own) {
              r_acc += (ve ? fabs(re) : 0.0) + (vo ? fabs(ro) : 0.0);
              d_acc += (le ? fabs(rh[k].x) : 0.0) + (lo ? fabs(rh[k].y) : 0.0);
              z.f[iz * P + j] = fe;
              z.f[iz * P + H + j] = fo;
            }
            F[s * P + j] = fe;
            F[s * P + H + j] = fo;
            U[s * P + j] = ve && !(iz & 1) ? fe * (c0 ? z.inv_e : z.inv_e2c) : 0.f;
            U[s * P + H + j] = vo && (iz & 1) ? fo * z.inv_e : 0.f;
          }
          below = here;
          here = nx[k];
        }
      }
    }
  }
  return make_double2(r_acc, d_acc);
}

// Level 0 down, a band a CTA: the residual; the other three colour sweeps,
// each on one row less; f of level 1; the band's own rows of u and f to z.u
// and z.f for the way up.  Psi stays as it is, so the last CTA to finish its
// sums decides here whether the solve is done: the WHILE node that holds the
// V-cycle runs on while `more` is set.
template <bool SM>
__global__ void __launch_bounds__(MG_NT, 1) k_mg_down0(const __grid_constant__ Mg0 z, const __grid_constant__ MgLevel C,
                                                       MgCall *call, cudaGraphConditionalHandle more, float *scratch,
                                                       size_t scratch_n)
{
  step_begin();
  if (call->skip) {
    if (blockIdx.x == 0 && threadIdx.x == 0)
      cudaGraphSetConditional(more, 0);
    return;
  }
  const int P = z.P, a0 = blockIdx.x * z.rp, b0 = min(a0 + z.rp, z.nz), r0 = a0 - MG_DOWN, n = b0 - a0 + 2 * MG_DOWN;
  float *U = band_buf<SM>(scratch, scratch_n), *F = U + (z.rp + 2 * MG_DOWN) * P;
  const double2 mine = resid0(z, call->Psi, call->rhs, call->umask, U, F, a0, b0);
  __shared__ bool last;
  {
    const double2 s = block_sums(mine.x, mine.y); // (its barrier also ends the residual)
    if (threadIdx.x == 0) {
      z.part[2 * blockIdx.x] = s.x;
      z.part[2 * blockIdx.x + 1] = s.y;
      __threadfence();
      last = atomicAdd(&call->ticket, 1u) == gridDim.x - 1;
    }
  }
  {
    Part0 t;
    part0(z, t, 0);
    for (int k = 1; k < 4; k++) { // colours 1, 0, 1
      relax0<false>(z, t, U, F, r0, k, n - k, k & 1);
      __syncthreads();
    }
    for (int s = MG_DOWN + (threadIdx.x >> 5); s < n - MG_DOWN; s += MG_W)
      for (int c0 = 4 * (threadIdx.x & 31); c0 < P; c0 += 128)
        st4(z.u + (size_t)(r0 + s) * P + c0, ld4(U + s * P + c0));
    relax0<true>(z, t, U, F, r0, MG_DOWN - 1, n - MG_DOWN + 1, 0);
    __syncthreads();
  }
  restrict0(C, P, F, r0, (a0 + C.cz - 1) / C.cz, min((b0 + C.cz - 1) / C.cz, C.Z), C.f);
  if (!last)
    return;
  __threadfence();
  double x = 0, y = 0; // the bands' sums, in a fixed order
  for (int k = threadIdx.x; k < (int)gridDim.x; k += MG_NT) {
    x += __ldcg(z.part + 2 * k);
    y += __ldcg(z.part + 2 * k + 1);
  }
  const double2 s = block_sums(x, y);
  if (threadIdx.x)
    return;
  const double total = s.x;
  if (call->cycles == 0)
    call->drive = call->rhs ? s.y : total; // poisson.c:40-43; a Laplace solve: its first residual
  const double drive = call->drive;
  const bool conv = total == 0 || total < call->accuracy * drive, stop = conv || call->cycles >= call->max_cycles;
  call->ticket = 0;
  cudaGraphSetConditional(more, !stop);
  if (!stop) {
    call->cycles++;
    return;
  }
  const long long result = conv ? call->cycles : -1;
  if (call->iters_out)
    *call->iters_out = result;
  if (call->st) {
    call->st->iterations = result;
    call->st->residual = total;
    call->st->driving = drive;
  }
  call->cnt->mg_cycles += call->cycles;
  call->cnt->sor_solves += 1;
}

// rows r0 .. r0+n-1 of a level's array g into the band buffer B (zero outside the array)
__device__ __forceinline__ void load9(const MgLevel &L, const float *g, float *B, int r0, int n)
{
  for (int s = threadIdx.x >> 5; s < n; s += MG_W) {
    const int I = r0 + s;
    const bool in = I >= 0 && I < L.Z;
    for (int c = 4 * (threadIdx.x & 31); c < L.P; c += 128)
      st4(B + s * L.P + c, in ? ldcg4(g + (size_t)(I + 1) * L.P + c) : make_float4(0.f, 0.f, 0.f, 0.f));
  }
}

__device__ __forceinline__ void store9(const MgLevel &L, float *g, const float *B, int r0, int Ia, int Ib)
{
  for (int I = Ia + (threadIdx.x >> 5); I < Ib; I += MG_W)
    for (int c = 4 * (threadIdx.x & 31); c < L.P; c += 128)
      st4(g + (size_t)(I + 1) * L.P + c, ld4(B + (I - r0) * L.P + c));
}

// A coarse level down, a band a CTA: two four-colour sweeps from u = 0, the
// halo shrinking by a row a row parity (the first needs none), then f of the
// next level from the residual of the band's rows.
template <bool SM, class Op>
__global__ void __launch_bounds__(MG_NT, 1) k_mg_down9(const __grid_constant__ MgLevel L,
                                                       const __grid_constant__ MgLevel C, float *scratch,
                                                       size_t scratch_n)
{
  float *buf = band_buf<SM>(scratch, scratch_n);
  const int I0 = blockIdx.x * L.rp, I1 = min(I0 + L.rp, L.Z), r0 = I0 - MG_DOWN, n = I1 - I0 + 2 * MG_DOWN;
  float *U = buf + L.P, *F = U + (L.rp + 2 * MG_DOWN + 1) * L.P; // a zero row on either side of U
  Op t;
  t.init(L, r0, r0, r0 + n);
  if (!SM) // (the scratch is the kernel's before)
    step_begin();
  for (int k = 4 * threadIdx.x; k < (n + 2) * L.P; k += 4 * MG_NT)
    st4(buf + k, make_float4(0.f, 0.f, 0.f, 0.f));
  if (SM)
    step_begin();
  load9(L, L.f, F, r0, n);
  __syncthreads();
  t.start(L, F);
#pragma unroll 1
  for (int k = 0; k < 4; k += 2) {
    rows9<0, 0>(L, t, U, F, r0, r0 + k, r0 + n - k);
    rows9<1, 0>(L, t, U, F, r0, r0 + k + 1, r0 + n - k - 1);
  }
  store9(L, L.u, U, r0, I0, I1);
  t.resid(L, U, F, F, r0, I0 - 1, I1 + 1);
  __syncthreads();
  restrict9(L, C, F, r0, (I0 + C.cz - 1) / C.cz, min((I1 + C.cz - 1) / C.cz, C.Z), C.f);
}

// A coarse level up: u of the way down plus the interpolated correction on
// the band and MG_UP halo rows, then two sweeps in the reverse colour order,
// into v.
template <bool SM, class Op>
__global__ void __launch_bounds__(MG_NT, 1) k_mg_up9(const __grid_constant__ MgLevel L, const __grid_constant__ MgLevel C,
                                                     float *scratch, size_t scratch_n)
{
  float *U = band_buf<SM>(scratch, scratch_n), *F = U + (L.rp + 2 * MG_DOWN) * L.P;
  const int I0 = blockIdx.x * L.rp, I1 = min(I0 + L.rp, L.Z), r0 = I0 - MG_UP, n = I1 - I0 + 2 * MG_UP;
  Op t;
  t.init(L, r0, r0, r0 + n);
  step_begin();
  load9(L, L.f, F, r0, n);
  load9(L, L.u, U, r0, n);
  __syncthreads();
  t.start(L, F);
  t.template prolong<true>(L, C, U, C.v, r0);
  __syncthreads();
#pragma unroll 1
  for (int k = 1; k < 4; k += 2) {
    rows9<1, 1>(L, t, U, F, r0, r0 + k, r0 + n - k);
    rows9<0, 1>(L, t, U, F, r0, r0 + k + 1, r0 + n - k - 1);
  }
  store9(L, L.v, U, r0, I0, I1);
}

// The bilinear correction from level C at the column pairs j .. j+3 (j a
// multiple of 4) of row i of level 0.
__device__ __forceinline__ void interp4(const MgLevel &C, int i, int j, float e[4], float o[4])
{
  const bool hz = C.cz == 2 && (i & 1); // a half-way row
  const float *p = C.v + (size_t)((C.cz == 2 ? i >> 1 : i) + 1) * C.P;
  float w[2][8];
#pragma unroll
  for (int h = 0; h < 2; h++, p += C.P)
    if (h == 0 || hz) {
      const float *x = p + 1 + (C.cr == 2 ? j >> 1 : j), *y = x + C.Q;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        w[h][k] = C.cr == 2 && k == 3 ? 0.f : __ldcg(x + k);
        w[h][4 + k] = C.cr == 2 && k > 1 ? 0.f : __ldcg(y + k);
      }
    }
#pragma unroll
  for (int h = 0; h < 2; h++)
    if (h == 0 || hz) {
      const float *v = w[h];
      float a[4], b[4]; // even and odd columns
      if (C.cr == 2) { // coarse nodes j .. j+4: v[0], v[4], v[1], v[5], v[2]
        a[0] = v[0], a[1] = v[4], a[2] = v[1], a[3] = v[5];
        b[0] = 0.5f * (v[0] + v[4]), b[1] = 0.5f * (v[4] + v[1]), b[2] = 0.5f * (v[1] + v[5]), b[3] = 0.5f * (v[5] + v[2]);
      } else {
#pragma unroll
        for (int k = 0; k < 4; k++)
          a[k] = v[k], b[k] = v[4 + k];
      }
#pragma unroll
      for (int k = 0; k < 4; k++) {
        e[k] = h ? 0.5f * e[k] + 0.5f * a[k] : a[k];
        o[k] = h ? 0.5f * o[k] + 0.5f * b[k] : b[k];
      }
    }
}

// Level 0 up: the same with colours 1, 0, 1, 0; the result goes to Psi in FP64.
template <bool SM>
__global__ void __launch_bounds__(MG_NT, 1) k_mg_up0(const __grid_constant__ Mg0 z, const __grid_constant__ MgLevel C,
                                                     const MgCall *call, float *scratch, size_t scratch_n)
{
  step_begin();
  const int P = z.P, H = P >> 1, K = (H / 4 + 31) >> 5, lane = threadIdx.x & 31;
  const float nan = __int_as_float(0x7fc00000);
  const int a0 = blockIdx.x * z.rp, b0 = min(a0 + z.rp, z.nz), r0 = a0 - MG_UP, n = b0 - a0 + 2 * MG_UP;
  float *U = band_buf<SM>(scratch, scratch_n), *F = U + (z.rp + 2 * MG_DOWN) * P;
  for (int t = threadIdx.x >> 5; t < n * K; t += MG_W) {
    const int s = (unsigned)t / (unsigned)K, j = 4 * ((t - s * K) * 32 + lane), iz = r0 + s;
    if (j >= H)
      continue;
    float4 f[2], u[2]; // even columns, odd columns
    f[0] = f[1] = make_float4(nan, nan, nan, nan);
    u[0] = u[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (iz >= z.lo && iz <= z.hi && 2 * j < z.cols) {
      const size_t at = (size_t)iz * P + j;
      f[0] = ldcg4(z.f + at);
      f[1] = ldcg4(z.f + at + H);
      u[0] = ldcg4(z.u + at);
      u[1] = ldcg4(z.u + at + H);
      float e[4], o[4];
      interp4(C, iz, j, e, o);
      u[0].x = f[0].x == f[0].x ? u[0].x + e[0] : 0.f;
      u[0].y = f[0].y == f[0].y ? u[0].y + e[1] : 0.f;
      u[0].z = f[0].z == f[0].z ? u[0].z + e[2] : 0.f;
      u[0].w = f[0].w == f[0].w ? u[0].w + e[3] : 0.f;
      u[1].x = f[1].x == f[1].x ? u[1].x + o[0] : 0.f;
      u[1].y = f[1].y == f[1].y ? u[1].y + o[1] : 0.f;
      u[1].z = f[1].z == f[1].z ? u[1].z + o[2] : 0.f;
      u[1].w = f[1].w == f[1].w ? u[1].w + o[3] : 0.f;
    }
    st4(U + s * P + j, u[0]);
    st4(U + s * P + H + j, u[1]);
    st4(F + s * P + j, f[0]);
    st4(F + s * P + H + j, f[1]);
  }
  {
    Part0 t;
    part0(z, t, 0);
    __syncthreads();
    for (int k = 1; k <= 4; k++) {
      relax0<false>(z, t, U, F, r0, k, n - k, k & 1);
      __syncthreads();
    }
  }
  double *Psi = call->Psi;
  const int K2 = (H + 31) >> 5, nt = (b0 - a0) * K2;
  for (int tb = threadIdx.x >> 5; tb < nt; tb += MG_W * MG_AHEAD) {
    double2 x[MG_AHEAD];
    int at[MG_AHEAD];
#pragma unroll
    for (int k = 0; k < MG_AHEAD; k++) {
      const int t = tb + k * MG_W, q = (unsigned)t / (unsigned)K2, j = (t - q * K2) * 32 + lane;
      at[k] = t < nt && 2 * j < z.cols ? (q + MG_UP) * P + j : -1;
      if (at[k] >= 0)
        x[k] = *reinterpret_cast<const double2 *>(Psi + node(a0 + q, 2 * j, P));
    }
#pragma unroll
    for (int k = 0; k < MG_AHEAD; k++)
      if (at[k] >= 0) {
        const int t = tb + k * MG_W, q = (unsigned)t / (unsigned)K2, j = (t - q * K2) * 32 + lane;
        const bool fe = F[at[k]] == F[at[k]], fo = F[at[k] + H] == F[at[k] + H];
        if (fe)
          x[k].x += (double)U[at[k]];
        if (fo)
          x[k].y += (double)U[at[k] + H];
        if (fe || fo)
          *reinterpret_cast<double2 *>(Psi + node(a0 + q, 2 * j, P)) = x[k];
      }
  }
}

// The coarsest level solved exactly: v = A^-1 f over its n unknowns (array
// indices idx[]), a warp a row of the inverse.  The rows (16 MB for 2048
// unknowns, from L2 or at worst in 3 us from HBM) are on their way to
// registers while f is gathered.  It takes the place of the V-cycle's levels
// below 2048 unknowns, whose kernel of one CTA was the longest of a cycle on
// all but the largest meshes, its sweeps being chains of CTA barriers: 34 -> 5.9
// us a cycle on a 3001 x 821 gun, 26 -> 4.3 on 1500 x 400, 24 -> 3.5 on 601 x
// 165; and an exact solve there saves cycles (6 -> 5 and 7 -> 5 of a cold start
// to 1e-6 on the first two).  Below about 2048 unknowns the inverse costs less
// to read than the two kernels of another level (5 us each).
__global__ void __launch_bounds__(MG_NT) k_mg_dense(const float *__restrict__ inv, int ld, const int *__restrict__ idx,
                                                    int n, const float *f, float *v)
{
  __shared__ __align__(16) float x[MG_MAX_DIRECT];
  constexpr int K = MG_MAX_DIRECT / 128;
  const int tid = threadIdx.x, lane = tid & 31, row = blockIdx.x * MG_W + (tid >> 5);
  float4 m[K];
  const float4 *src = reinterpret_cast<const float4 *>(inv + (size_t)min(row, n - 1) * ld) + lane;
#pragma unroll
  for (int k = 0; k < K; k++)
    m[k] = 128 * k < ld ? __ldg(src + 32 * k) : make_float4(0.f, 0.f, 0.f, 0.f);
  const int at = __ldg(idx + min(row, n - 1));
  step_begin();
  for (int i = tid; i < ld; i += MG_NT)
    x[i] = i < n ? __ldcg(f + __ldg(idx + i)) : 0.f;
  __syncthreads();
  float acc = 0.f;
#pragma unroll
  for (int k = 0; k < K; k++)
    if (128 * k < ld) {
      const float4 y = ld4(x + 4 * (32 * k + lane));
      acc += m[k].x * y.x + m[k].y * y.y + (m[k].z * y.z + m[k].w * y.w);
    }
  for (int o = 16; o > 0; o >>= 1)
    acc += __shfl_down_sync(0xffffffffu, acc, o);
  if (lane == 0 && row < n)
    v[at] = acc;
}

// The inverse's columns from the banded factors (rows of 2 b + 1 doubles: L
// below the unit diagonal, 1 / U's diagonal, U above it): a warp takes
// MG_INV_COLS columns through the forward and the backward substitution, four
// lanes a column with every fourth coupling each.  The columns stay in shared
// memory (128 KB for 2048 unknowns) from the first pass to the end: a copy in
// global memory would be twice the inverse's own size for the time of the
// set-up, and an instance's largest need of memory.  Each row is a chain
// (product, sum over the lanes, the next row's read of it), so the factors' rows
// come MG_INV_AHEAD rows ahead of their use.  A gun's set-up: 0.36 ms on 90 x 90,
// 0.64 on 424 x 232, 0.87 on 3001 x 821; with the columns in global memory, 32 a
// warp and a lane a column, 1.0, 2.0 and 3.0.
constexpr int MG_INV_COLS = 8, MG_INV_AHEAD = 6;
__host__ __device__ inline size_t mg_inverse_smem(int n, int b)
{
  return ((size_t)n * MG_INV_COLS + (size_t)MG_INV_AHEAD * (b + 1)) * sizeof(double);
}

__global__ void __launch_bounds__(32) k_mg_inverse(int n, int b, const double *__restrict__ lu, float *inv, int ld)
{
  extern __shared__ double y[]; // n x MG_INV_COLS; then the rows ahead, b + 1 doubles each
  const int lane = threadIdx.x, col = lane & (MG_INV_COLS - 1), q = lane / MG_INV_COLS;
  const int c0 = MG_INV_COLS * blockIdx.x, c = c0 + col, w = 2 * b + 1;
  if (c0 >= n) { // padding
    for (int i = q; i < n; i += 4)
      inv[(size_t)i * ld + c] = 0.f;
    return;
  }
  double *rows = y + (size_t)n * MG_INV_COLS;
  // row i's b + 1 entries from its at-th on, to place `to` (no row: an empty group)
  auto fetch = [&](int i, int at, int to) {
    if (i >= 0 && i < n)
      for (int k = lane; k <= b; k += 32)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(rows + to * (b + 1) + k)),
                     "l"(lu + (size_t)i * w + at + k)
                     : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto arrived = [&]() { // the oldest of the rows ahead
    asm volatile("cp.async.wait_group %0;" ::"n"(MG_INV_AHEAD - 2) : "memory");
    __syncwarp();
  };
  auto total = [](double acc) { // of the column's four lanes
    acc += __shfl_xor_sync(0xffffffffu, acc, MG_INV_COLS);
    return acc + __shfl_xor_sync(0xffffffffu, acc, 2 * MG_INV_COLS);
  };
  for (int k = 0; k < MG_INV_AHEAD - 1; k++)
    fetch(c0 + k, 0, k);
  for (int i = c0, r = 0; i < n; i++, r = r == MG_INV_AHEAD - 1 ? 0 : r + 1) { // (zero before)
    arrived();
    fetch(i + MG_INV_AHEAD - 1, 0, r == 0 ? MG_INV_AHEAD - 1 : r - 1);
    const double *l = rows + r * (b + 1) + b; // l[-k]: the coupling to row i - k
    double acc = q == 0 && i == c ? 1.0 : 0.0;
    const int last = min(b, i - c0);
#pragma unroll 4
    for (int k = 1 + q; k <= last; k += 4)
      acc -= l[-k] * y[(i - k) * MG_INV_COLS + col];
    acc = total(acc);
    if (q == 0)
      y[i * MG_INV_COLS + col] = acc;
    __syncwarp();
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncwarp();
  for (int k = 0; k < MG_INV_AHEAD - 1; k++)
    fetch(n - 1 - k, b, k);
  for (int i = n - 1, r = 0; i >= 0; i--, r = r == MG_INV_AHEAD - 1 ? 0 : r + 1) {
    arrived();
    fetch(i - MG_INV_AHEAD + 1, b, r == 0 ? MG_INV_AHEAD - 1 : r - 1);
    const double *u = rows + r * (b + 1); // u[k]: the coupling to row i + k
    double acc = q == 0 && i >= c0 ? y[i * MG_INV_COLS + col] : 0.0;
    const int last = min(b, n - 1 - i);
#pragma unroll 4
    for (int k = 1 + q; k <= last; k += 4)
      acc -= u[k] * y[(i + k) * MG_INV_COLS + col];
    const double x = total(acc) * u[0];
    if (q == 0) {
      y[i * MG_INV_COLS + col] = x;
      inv[(size_t)i * ld + c] = (float)x;
    }
    __syncwarp();
  }
}

// A coarsest level that has no inverse (one that cannot be coarsened further
// with more unknowns than MG_MAX_DIRECT): sweeps by one CTA.  With SM u and f
// lie in shared memory, else in global memory.  The result goes to v.
template <bool SM, class Op> __global__ void __launch_bounds__(MG_NT, 1) k_mg_coarse(const __grid_constant__ MgLevel L)
{
  step_begin();
  const int tid = threadIdx.x, n = (L.Z + 2) * L.P;
  float *u = SM ? reinterpret_cast<float *>(mg_smem) : L.u, *f = SM ? u + n : L.f; // row -1 first
  for (int k = 4 * tid; k < n; k += 4 * MG_NT) {
    st4(u + k, make_float4(0.f, 0.f, 0.f, 0.f));
    if (SM)
      st4(f + k, ldcg4(L.f + k));
  }
  __syncthreads();
  Op t;
  t.init(L, -1, 0, L.Z);
  t.start(L, f);
#pragma unroll 1
  for (int k = 0; k < MG_COARSE_SWEEPS; k++) {
    rows9<0, 0>(L, t, u, f, -1, 0, L.Z);
    rows9<1, 0>(L, t, u, f, -1, 0, L.Z);
  }
  for (int k = 4 * tid; k < n; k += 4 * MG_NT)
    st4(L.v + k, ld4(u + k));
}

// ---- host: the level hierarchy

// fn(lo, hi) over [0, n) in contiguous chunks on up to 16 host threads (the
// hierarchy of a 2.5M-node mesh takes over half a second on one core)
template <class Fn>
void parallel_rows(int n, Fn fn)
{
  const int nt = std::max(1, std::min({16, (int)std::thread::hardware_concurrency(), n / 8}));
  if (nt <= 1) {
    fn(0, n);
    return;
  }
  std::vector<std::thread> pool;
  const int chunk = (n + nt - 1) / nt;
  for (int t = 0; t < nt; t++) {
    const int lo = t * chunk, hi = std::min(n, lo + chunk);
    if (lo >= hi)
      continue;
    try {
      pool.emplace_back(fn, lo, hi);
    } catch (const std::system_error &) {
      fn(lo, hi); // no thread to be had: this chunk on the caller's thread
    }
  }
  for (std::thread &th : pool)
    th.join();
}

// level-0 operator as nine-point rows (only the five-point entries are
// nonzero): coefficient of node (iz+dz, ir+dr) at k = (dz+1)*3 + (dr+1)
struct Stencil {
  int Z = 0, R = 0;
  std::vector<double> c; // [9][Z*R]
  std::vector<uint8_t> unk;
  double &at(int k, int i, int j) { return c[(size_t)k * Z * R + (size_t)i * R + j]; }
  double at(int k, int i, int j) const { return c[(size_t)k * Z * R + (size_t)i * R + j]; }
};

void fine_stencil(const DevMesh &m, const int16_t *flags, int lo, int hi, Stencil &S)
{
  const int nz = m.nz, nr = m.nr, cols = nr - 1;
  S.Z = nz + 1;
  S.R = nr + 1;
  S.c.assign((size_t)9 * S.Z * S.R, 0.0);
  S.unk.assign((size_t)S.Z * S.R, 0);
  for (int iz = lo; iz <= hi; iz++)
    for (int ir = 0; ir < cols; ir++)
      if (!(flags[(size_t)iz * (nr + 1) + ir] & (SPIFFE_FL_IS_SURFACE | SPIFFE_FL_IS_INSIDE)))
        S.unk[(size_t)iz * S.R + ir] = 1;
  const double a = 1 / (m.dz * m.dz), dr2 = m.dr * m.dr;
  const double e = -2 * (1 / (m.dz * m.dz) + 1 / dr2);
  // each node writes only its own stencil row
  parallel_rows(hi - lo + 1, [&](int r0, int r1) {
  for (int iz = lo + r0; iz < lo + r1; iz++)
    for (int ir = 0; ir < cols; ir++) {
      if (!S.unk[(size_t)iz * S.R + ir])
        continue;
      double cu = a, cd = a;
      int zu = iz + 1, zd = iz - 1;
      if (iz == 0 && lo == 0) { // mirrored end rows (poisson.c:67-84, :102-118)
        zd = iz + 1;
      } else if (iz == nz - 1 && hi == nz - 1) {
        zu = iz - 1;
      }
      double cr, cl, dg;
      if (ir == 0) {
        cr = 4 / dr2;
        cl = 0;
        dg = e - 2 / dr2;
      } else {
        cr = 1 / dr2 * (1 + 1. / (2 * ir));
        cl = 1 / dr2 * (1 - 1. / (2 * ir));
        dg = e;
      }
      auto add = [&](int z2, int r2, double v) {
        if (v == 0 || z2 < 0 || z2 >= S.Z || r2 < 0 || r2 >= S.R || !S.unk[(size_t)z2 * S.R + r2])
          return;
        S.at((z2 - iz + 1) * 3 + (r2 - ir + 1), iz, ir) += v;
      };
      add(zu, ir, cu);
      add(zd, ir, cd);
      add(iz, ir + 1, cr);
      add(iz, ir - 1, cl);
      S.at(4, iz, ir) = dg;
    }
  });
}

// annulus weight of column j of a level of spacing 1 (the axis node: 1/8)
inline double vol(int j) { return j ? (double)j : 0.125; }

// Galerkin R A P from level F to C (nodes cz I, cr J of F: cz, cr = 2 to
// coarsen a direction, 1 to keep it); restriction weights rw[J][3] for F
// columns cr J - 1, cr J, cr J + 1 (with cz = 2 the z weights 1/2, 1, 1/2
// apply on top)
void galerkin(const Stencil &F, Stencil &C, std::vector<double> &rw, int cz, int cr)
{
  C.Z = cz == 2 ? (F.Z + 1) / 2 : F.Z;
  C.R = cr == 2 ? (F.R + 1) / 2 : F.R;
  C.c.assign((size_t)9 * C.Z * C.R, 0.0);
  C.unk.assign((size_t)C.Z * C.R, 0);
  for (int I = 0; I < C.Z; I++)
    for (int J = 0; J < C.R; J++)
      C.unk[(size_t)I * C.R + J] = F.unk[(size_t)(cz * I) * F.R + cr * J];
  rw.assign((size_t)3 * C.R, 0.0);
  for (int J = 0; J < C.R; J++)
    for (int dj = -1; dj <= 1; dj++) {
      const int j = cr * J + dj;
      if (j < 0 || j >= F.R || (cr == 1 && dj))
        continue;
      // in fine units: coarse spacing 2, Vc(J) = 2 vc with vc = 2J (axis:
      // 1/4); coarse spacing 1, Vc(J) = vol(J) = 2 vc
      const double vc = cr == 2 ? (J ? 2.0 * J : 0.25) : 0.5 * vol(J);
      rw[(size_t)3 * J + dj + 1] = (dj ? 0.5 : 1.0) * vol(j) / (4 * vc);
    }
  auto cunk = [&](int I, int J) { return I >= 0 && I < C.Z && J >= 0 && J < C.R && C.unk[(size_t)I * C.R + J]; };
  // coarse rows in parallel: each node writes only its own stencil and flag,
  // and reads the neighbours' flags as they were before any hold below (a
  // coupling to a node held here is removed by the pass after, so the
  // stencils do not depend on the order the rows are done in)
  const std::vector<uint8_t> unk0 = C.unk;
  auto cunk0 = [&](int I, int J) { return I >= 0 && I < C.Z && J >= 0 && J < C.R && unk0[(size_t)I * C.R + J]; };
  parallel_rows(C.Z, [&](int I0, int I1) {
  for (int I = I0; I < I1; I++)
    for (int J = 0; J < C.R; J++) {
      if (!C.unk[(size_t)I * C.R + J])
        continue;
      double acc[9] = {0};
      const int dz0 = cz == 2 ? -1 : 0, dr0 = cr == 2 ? -1 : 0;
      for (int di = dz0; di <= -dz0; di++)
        for (int dj = dr0; dj <= -dr0; dj++) {
          const int i = cz * I + di, j = cr * J + dj;
          if (i < 0 || i >= F.Z || j < 0 || j >= F.R || !F.unk[(size_t)i * F.R + j])
            continue;
          const double r = (di ? 0.5 : 1.0) * rw[(size_t)3 * J + dj + 1];
          for (int k = 0; k < 9; k++) {
            const double v = F.at(k, i, j);
            if (v == 0)
              continue;
            const int ni = i + k / 3 - 1, nj = j + k % 3 - 1; // an unknown fine node
            // its coarse parents (bilinear interpolation; along a direction
            // kept, the node itself)
            const bool hz = cz == 2 && (ni & 1), hr = cr == 2 && (nj & 1);
            const int pz0 = cz == 2 ? ni >> 1 : ni, pr0 = cr == 2 ? nj >> 1 : nj;
            const int nzp = hz ? 2 : 1, nrp = hr ? 2 : 1;
            const double wz = hz ? 0.5 : 1.0, wr = hr ? 0.5 : 1.0;
            for (int pz = 0; pz < nzp; pz++)
              for (int pr = 0; pr < nrp; pr++) {
                const int K = pz0 + pz, Lc = pr0 + pr;
                if (!cunk0(K, Lc))
                  continue;
                acc[(K - I + 1) * 3 + (Lc - J + 1)] += r * v * wz * wr;
              }
          }
        }
      for (int k = 0; k < 9; k++)
        C.at(k, I, J) = acc[k];
      if (!(acc[4] < 0)) { // not a proper diagonal: hold the node
        C.unk[(size_t)I * C.R + J] = 0;
        for (int k = 0; k < 9; k++)
          C.at(k, I, J) = 0;
      }
    }
  });
  // couplings to nodes that were held above (after every row's hold)
  parallel_rows(C.Z, [&](int I0, int I1) {
    for (int I = I0; I < I1; I++)
      for (int J = 0; J < C.R; J++)
        for (int k = 0; k < 9; k++)
          if (C.at(k, I, J) != 0 && !cunk(I + k / 3 - 1, J + k % 3 - 1))
            C.at(k, I, J) = 0;
  });
}

size_t unknowns(const Stencil &S)
{
  size_t n = 0;
  for (uint8_t u : S.unk)
    n += u;
  return n;
}

} // namespace

extern "C" void s32_mg_free(Mg32Work *w)
{
  if (w->exec)
    cudaGraphExecDestroy((cudaGraphExec_t)w->exec);
  dev_free(w->mem);
  *w = Mg32Work();
}

namespace {
// The coarsest level's operator over its unknowns as banded LU factors, for
// k_mg_inverse; false when the level has more than MG_MAX_DIRECT unknowns or
// couplings beyond MG_MAX_BAND, or a pivot is not negative.  No pivoting: the
// operator is negative definite in the annulus-weighted inner product, and a
// Galerkin product keeps that.  The unknowns are numbered along the shorter
// direction, so the band is that direction's length.
bool coarse_factor(const Stencil &S, const MgLevel &D, std::vector<double> &lu, int &b, std::vector<int> &idx)
{
  std::vector<int> num((size_t)S.Z * S.R, -1);
  idx.clear();
  const bool rows = S.R <= S.Z;
  for (int p = 0; p < (rows ? S.Z : S.R); p++)
    for (int q = 0; q < (rows ? S.R : S.Z); q++) {
      const int I = rows ? p : q, J = rows ? q : p;
      if (S.unk[(size_t)I * S.R + J]) {
        num[(size_t)I * S.R + J] = (int)idx.size();
        idx.push_back((I + 1) * D.P + (J & 1) * D.Q + (J >> 1) + 1);
      }
    }
  const int n = (int)idx.size();
  if (n == 0 || n > MG_MAX_DIRECT)
    return false;
  auto couplings = [&](auto fn) {
    for (int I = 0; I < S.Z; I++)
      for (int J = 0; J < S.R; J++) {
        const int r = num[(size_t)I * S.R + J];
        for (int k = 0; r >= 0 && k < 9; k++) {
          const int i2 = I + k / 3 - 1, j2 = J + k % 3 - 1;
          if (i2 < 0 || i2 >= S.Z || j2 < 0 || j2 >= S.R)
            continue;
          const int c = num[(size_t)i2 * S.R + j2];
          if (c >= 0)
            fn(r, c, S.at(k, I, J));
        }
      }
  };
  b = 1;
  couplings([&](int r, int c, double) { b = std::max(b, std::abs(r - c)); });
  if (b > MG_MAX_BAND)
    return false;
  const int w = 2 * b + 1;
  lu.assign((size_t)n * w, 0.0); // (r, c) at r w + b + c - r
  couplings([&](int r, int c, double v) { lu[(size_t)r * w + b + c - r] += v; });
  for (int k = 0; k < n; k++) {
    double *pk = lu.data() + (size_t)k * w + b; // pk[j]: (k, k + j)
    if (!(pk[0] < 0))
      return false;
    pk[0] = 1 / pk[0];
    const int last = std::min(b, n - 1 - k);
    for (int i = 1; i <= last; i++) {
      double *pi = lu.data() + (size_t)(k + i) * w + b - i; // pi[j]: (k + i, k + j)
      if (pi[0] == 0)
        continue;
      const double m = pi[0] *= pk[0];
      for (int j = 1; j <= last; j++)
        pi[j] -= m * pk[j];
    }
  }
  return true;
}
} // namespace

namespace {
// the kernels whose bands lie in shared memory
std::vector<const void *> mg_smem_kernels()
{
  return {(const void *)k_mg_down0<true>,          (const void *)k_mg_up0<true>,
          (const void *)k_mg_down9<true, Fix9<1>>, (const void *)k_mg_down9<true, Fix9<2>>,
          (const void *)k_mg_down9<true, Run9>,    (const void *)k_mg_up9<true, Fix9<1>>,
          (const void *)k_mg_up9<true, Fix9<2>>,   (const void *)k_mg_up9<true, Run9>,
          (const void *)k_mg_coarse<true, Fix9<2>>};
}

// the coarsest level's inverse and its unknowns' array indices, on the device
struct MgDense {
  const float *inv;
  const int *idx;
  int n, ld;
};

// The solve as a graph: the residual's kernel, then a WHILE node around a
// V-cycle that ends with the next residual.
int mg_graph(Mg32Work *w, Mg0 z, int last, bool sm, const MgDense *dense, bool coarse_sm, float *scratch, size_t budget)
{
  MgLevel *lev = w->lev;
  MgCall *call = (MgCall *)w->call;
  auto bytes_of = [&](int rp, int P) { return sm ? (size_t)(2 * rp + 4 * MG_DOWN + 2) * P * sizeof(float) : 0; };
  auto floats_of = [](int rp, int P) { return (size_t)(2 * rp + 4 * MG_DOWN + 2) * P; };
  const void *kd0 = sm ? (const void *)k_mg_down0<true> : (const void *)k_mg_down0<false>;
  // pairs of a row parity in n rows, a thread's number of them: Fix9 or Run9
  auto pairs = [](const MgLevel &D, int n) { return (size_t)((n + 1) / 2) * ((D.R + 1) / 2); };
  auto kd9 = [&](const MgLevel &D) {
    const size_t n = pairs(D, D.rp + 2 * MG_DOWN);
    return !sm                ? (const void *)k_mg_down9<false, Run9>
           : n <= MG_NT       ? (const void *)k_mg_down9<true, Fix9<1>>
           : n <= 2 * MG_NT   ? (const void *)k_mg_down9<true, Fix9<2>>
                              : (const void *)k_mg_down9<true, Run9>;
  };
  auto ku9 = [&](const MgLevel &D) {
    const size_t n = pairs(D, D.rp + 2 * MG_UP);
    return !sm                ? (const void *)k_mg_up9<false, Run9>
           : n <= MG_NT       ? (const void *)k_mg_up9<true, Fix9<1>>
           : n <= 2 * MG_NT   ? (const void *)k_mg_up9<true, Fix9<2>>
                              : (const void *)k_mg_up9<true, Run9>;
  };
  const void *ku0 = sm ? (const void *)k_mg_up0<true> : (const void *)k_mg_up0<false>;
  const bool coarse_fix = coarse_sm && pairs(lev[last], lev[last].Z) <= 2 * MG_NT;
  const void *kc = coarse_fix ? (const void *)k_mg_coarse<true, Fix9<2>> : (const void *)k_mg_coarse<false, Run9>;
  cudaError_t e = cudaSuccess;
  // the attribute is process-wide: the kernels' limit, not this instance's need
  for (const void *k : mg_smem_kernels())
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)budget);
  cudaGraph_t graph = nullptr;
  if (e == cudaSuccess)
    e = cudaGraphCreate(&graph, 0);
  if (e != cudaSuccess)
    return (int)e;
  cudaGraphConditionalHandle more{};
  e = cudaGraphConditionalHandleCreate(&more, graph, 0, 0);
  cudaGraphNode_t prev = nullptr;
  auto add = [&](cudaGraph_t g, const void *k, int blocks, size_t smem, void **args) {
    if (e != cudaSuccess)
      return;
    cudaKernelNodeParams p{};
    p.func = (void *)k;
    p.gridDim = dim3(blocks);
    p.blockDim = dim3(MG_NT);
    p.sharedMemBytes = (unsigned)smem;
    p.kernelParams = args;
    cudaGraphNode_t n;
    e = cudaGraphAddKernelNode(&n, g, nullptr, 0, &p);
    if (e == cudaSuccess && prev) { // begins while the one before ends (step_begin)
      cudaGraphEdgeData next{};
      next.from_port = cudaGraphKernelNodePortProgrammatic;
      next.type = cudaGraphDependencyTypeProgrammatic;
      e = cudaGraphAddDependencies_v2(g, &prev, &n, &next, 1);
    }
    prev = n;
  };
  size_t n0 = floats_of(z.rp, z.P);
  void *a_down0[] = {&z, &lev[1], &call, &more, &scratch, &n0};
  void *a_up0[] = {&z, &lev[1], &call, &scratch, &n0};
  add(graph, kd0, z.nb, bytes_of(z.rp, z.P), a_down0);
  cudaGraphNodeParams cp{};
  cp.type = cudaGraphNodeTypeConditional;
  cp.conditional.handle = more;
  cp.conditional.type = cudaGraphCondTypeWhile;
  cp.conditional.size = 1;
  cudaGraphNode_t loop;
  if (e == cudaSuccess)
    e = cudaGraphAddNode(&loop, graph, &prev, 1, &cp);
  if (e == cudaSuccess) {
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    prev = nullptr;
    for (int l = 1; l < last; l++) {
      size_t n = floats_of(lev[l].rp, lev[l].P);
      void *a9[] = {&lev[l], &lev[l + 1], &scratch, &n};
      add(body, kd9(lev[l]), lev[l].nb, bytes_of(lev[l].rp, lev[l].P), a9);
    }
    const MgLevel &C = lev[last];
    if (dense) {
      MgDense d = *dense;
      void *ad[] = {&d.inv, &d.ld, &d.idx, &d.n, (void *)&C.f, (void *)&C.v};
      add(body, (const void *)k_mg_dense, (d.n + MG_W - 1) / MG_W, 0, ad);
    } else {
      void *ac[] = {&lev[last]};
      add(body, kc, 1, coarse_fix ? 2 * sizeof(float) * (size_t)(C.Z + 2) * C.P : 0, ac);
    }
    for (int l = last - 1; l >= 1; l--) {
      size_t n = floats_of(lev[l].rp, lev[l].P);
      void *a9[] = {&lev[l], &lev[l + 1], &scratch, &n};
      add(body, ku9(lev[l]), lev[l].nb, bytes_of(lev[l].rp, lev[l].P), a9);
    }
    add(body, ku0, z.nb, bytes_of(z.rp, z.P), a_up0);
    add(body, kd0, z.nb, bytes_of(z.rp, z.P), a_down0);
  }
  cudaGraphExec_t exec = nullptr;
  if (e == cudaSuccess)
    e = cudaGraphInstantiate(&exec, graph, 0);
  w->exec = exec;
  cudaGraphDestroy(graph);
  return (int)e;
}
} // namespace

extern "C" int s32_mg_setup(const DevMesh *m, const int16_t *flags, Mg32Work *w, cudaStream_t s)
{
  s32_mg_free(w);
  const int lo = m->left_bc == SPIFFE_DIRICHLET ? 0 : 1;
  const int hi = m->right_bc == SPIFFE_DIRICHLET ? m->nz - 1 : m->nz - 2;
  std::vector<Stencil> lev(1);
  std::vector<std::vector<double>> rws(1);
  fine_stencil(*m, flags, lo, hi, lev[0]);
  // Semi-coarsening: where the spacing in one direction is at least twice
  // the other's, the operator couples nodes far more strongly along the
  // finer direction, point Gauss-Seidel smooths the error only along it,
  // and only that direction is coarsened (on a 165 x 357 gun mesh with
  // dz = 8 dr, 64 V-cycles a correction with both directions coarsened).
  std::vector<int> czs(1, 2), crs(1, 2);
  double sz = m->dz, sr = m->dr; // the finest level's spacings so far
  while ((int)lev.size() < MG_MAX_LEVELS) {
    const Stencil &F = lev.back();
    if (unknowns(F) <= (size_t)(lev.size() > 1 ? MG_MAX_DIRECT : MG_MIN_UNKNOWNS))
      break;
    const int cz = sz >= 2 * sr ? 1 : 2, cr = sr >= 2 * sz ? 1 : 2;
    if ((cz == 2 && F.Z < 5) || (cr == 2 && F.R < 5))
      break;
    Stencil C;
    std::vector<double> rw;
    galerkin(F, C, rw, cz, cr);
    if (unknowns(C) == 0)
      break;
    lev.push_back(std::move(C));
    rws.push_back(std::move(rw));
    czs.push_back(cz);
    crs.push_back(cr);
    sz *= cz;
    sr *= cr;
  }
  const int L = (int)lev.size();
  if (L < 2)
    return (int)cudaErrorInvalidConfiguration; // a mesh too small to coarsen: the caller uses SOR
  // constant data, gathered on the host and copied once: the coefficients of
  // each level's distinct rows (a row's metal decides them, so a gun has few;
  // cls names a row's), the restriction weights, level 0's radial couplings
  const int P0 = m->pitch;
  std::vector<char> blob;
  auto put = [&](const void *p, size_t n) {
    const size_t at = blob.size();
    blob.resize((at + n + 255) / 256 * 256);
    std::memcpy(blob.data() + at, p, n);
    return at;
  };
  std::vector<size_t> coff(L), roff(L), ioff(L);
  for (int l = 1; l < L; l++) {
    const Stencil &S = lev[l];
    MgLevel &D = w->lev[l];
    D.Z = S.Z;
    D.R = S.R;
    D.cz = czs[l];
    D.cr = crs[l];
    D.Q = ((S.R >> 1) + 2 + 15) / 16 * 16;
    D.P = 2 * D.Q;
    const size_t row_n = (size_t)MG_NCOEF * D.P;
    std::vector<float> all((size_t)S.Z * row_n, 0.f);
    parallel_rows(S.Z, [&](int I0, int I1) {
      for (int I = I0; I < I1; I++) {
        float *row = all.data() + (size_t)I * row_n;
        for (int J = 0; J < S.R; J++) {
          if (!S.unk[(size_t)I * S.R + J])
            continue;
          const int at = (J & 1) * D.Q + (J >> 1) + 1;
          const double dg = S.at(4, I, J);
          int q = 0;
          for (int k = 0; k < 9; k++)
            if (k != 4)
              row[(size_t)D.P * q++ + at] = (float)(S.at(k, I, J) / dg);
          row[(size_t)D.P * MG_INVD + at] = (float)(1 / dg);
          row[(size_t)D.P * MG_DIAG + at] = (float)dg;
        }
      }
    });
    // a row's class: most rows are like the one before
    std::vector<uint8_t> same(S.Z, 0);
    parallel_rows(S.Z, [&](int I0, int I1) {
      for (int I = std::max(I0, 1); I < I1; I++)
        same[I] = !std::memcmp(all.data() + (size_t)I * row_n, all.data() + (size_t)(I - 1) * row_n, row_n * sizeof(float));
    });
    std::unordered_multimap<uint64_t, int> seen; // hash -> class
    std::vector<int> cls(S.Z), first;            // a row's class, a class's first row
    for (int I = 0; I < S.Z; I++) {
      const float *row = all.data() + (size_t)I * row_n;
      int c = same[I] ? cls[I - 1] : -1;
      if (c < 0) {
        uint64_t h = 1469598103934665603ull; // FNV-1a over 32-bit words
        for (size_t k = 0; k < row_n; k++) {
          uint32_t b;
          std::memcpy(&b, row + k, 4);
          h = (h ^ b) * 1099511628211ull;
        }
        const auto range = seen.equal_range(h);
        for (auto it = range.first; it != range.second && c < 0; ++it)
          if (!std::memcmp(all.data() + (size_t)first[it->second] * row_n, row, row_n * sizeof(float)))
            c = it->second;
        if (c < 0) {
          c = (int)first.size();
          first.push_back(I);
          seen.emplace(h, c);
        }
      }
      cls[I] = c;
    }
    std::vector<float> packed(first.size() * row_n);
    for (size_t c = 0; c < first.size(); c++)
      std::memcpy(packed.data() + c * row_n, all.data() + (size_t)first[c] * row_n, row_n * sizeof(float));
    coff[l] = put(packed.data(), packed.size() * sizeof(float));
    ioff[l] = put(cls.data(), cls.size() * sizeof(int));
    std::vector<float> rw(rws[l].begin(), rws[l].end());
    roff[l] = put(rw.data(), rw.size() * sizeof(float));
  }
  std::vector<float> crow(P0, 0.f), drow(P0, 0.f);
  std::vector<double> cpd(P0, 0.0), cmd(P0, 0.0);
  const double dr2_inv = 1 / (m->dr * m->dr);
  for (int ir = 0; ir <= m->nr; ir++) {
    const double h = ir ? 0.5 / ir : 0;
    cpd[ir] = ir ? dr2_inv * (1 + h) : 4 / (m->dr * m->dr);
    cmd[ir] = ir ? dr2_inv * (1 - h) : 0;
    crow[ir] = (float)cpd[ir]; // the axis node has no inner neighbour
    drow[ir] = (float)cmd[ir];
  }
  const size_t o_crow = put(crow.data(), P0 * sizeof(float)), o_drow = put(drow.data(), P0 * sizeof(float));
  const size_t o_cpd = put(cpd.data(), P0 * sizeof(double)), o_cmd = put(cmd.data(), P0 * sizeof(double));
  std::vector<double> lu;
  std::vector<int> cidx;
  int band_b = 0;
  size_t o_cidx = 0;
  const bool direct = coarse_factor(lev[L - 1], w->lev[L - 1], lu, band_b, cidx);
  const int cn = (int)cidx.size(), ld = (cn + 127) / 128 * 128;
  if (direct)
    o_cidx = put(cidx.data(), cidx.size() * sizeof(int));
  const int last = L - 1;

  // Bands: a level's rows in one band per SM at most, and no more of them than
  // the mesh gives work (a small mesh's solve leaves the other SMs to other
  // instances' kernels; each band recomputes its halo), of MG_MIN_ROWS rows at
  // least; shorter ones where a band of u and f with its halos would not fit
  // shared memory.  A mesh whose row is too long for MG_MIN_ROWS of them keeps
  // its bands in global memory.
  int dev = 0, sms = 0, max_smem = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  const size_t mesh_nodes = (size_t)(m->nz + 1) * (m->nr + 1);
  const int grid = (int)std::min<size_t>((size_t)sms, std::max<size_t>(1, (mesh_nodes + MG_NODES_PER_CTA - 1) / MG_NODES_PER_CTA));
  size_t fixed = 0; // the kernels' own shared memory
  for (const void *k : mg_smem_kernels()) {
    cudaFuncAttributes fa{};
    const cudaError_t e = cudaFuncGetAttributes(&fa, k);
    if (e != cudaSuccess)
      return (int)e;
    fixed = std::max(fixed, fa.sharedSizeBytes);
  }
  const size_t budget = ((size_t)max_smem - fixed) / sizeof(float);
  auto band_n = [](int rp, int P) { return (size_t)(2 * rp + 4 * MG_DOWN + 2) * P; };
  bool fits = true;
  size_t need = 0; // floats of the largest band
  auto band = [&](int rows, int P, int &rp, int &nb) {
    rp = std::max((rows + grid - 1) / grid, std::min(MG_MIN_ROWS, rows));
    if (band_n(rp, P) > budget && band_n(MG_MIN_ROWS, P) <= budget)
      rp = (int)((budget / P - 4 * MG_DOWN - 2) / 2);
    nb = (rows + rp - 1) / rp;
    fits = fits && band_n(rp, P) <= budget;
    need = std::max(need, band_n(rp, P) * nb);
  };
  int rp0 = 0, nb0 = 0;
  band(m->nz, P0, rp0, nb0);
  for (int l = 1; l < last; l++)
    band(w->lev[l].Z, w->lev[l].P, w->lev[l].rp, w->lev[l].nb);
  const bool coarse_fits = 2 * (size_t)(lev[last].Z + 2) * w->lev[last].P <= budget;

  // device memory, one block: the constant data, level 0's u0 and f0 at the
  // mesh pitch, each coarse level's u, f and v of (Z+2) x P floats, the
  // bands' global buffers where they are needed, sums and barrier words
  const size_t n0 = (size_t)(m->nz + 1) * P0;
  size_t bytes = blob.size();
  const size_t o_u0 = bytes;
  bytes += 2 * n0 * sizeof(float);
  std::vector<size_t> off(L);
  for (int l = 1; l < L; l++) {
    off[l] = bytes;
    bytes += (size_t)3 * (lev[l].Z + 2) * w->lev[l].P * sizeof(float);
  }
  const size_t o_scratch = bytes;
  bytes += fits ? 0 : need * sizeof(float);
  const size_t o_part = bytes;
  bytes += ((size_t)2 * nb0 * sizeof(double) + 255) / 256 * 256;
  const size_t o_call = bytes;
  bytes += (sizeof(MgCall) + 255) / 256 * 256;
  const size_t o_inv = bytes;
  bytes += direct ? (size_t)cn * ld * sizeof(float) : 0;
  char *mem = nullptr;
  cudaError_t e = dev_malloc(&mem, bytes);
  if (e != cudaSuccess)
    return (int)e;
  w->mem = mem;
  w->bytes = bytes;
  w->call = mem + o_call;
  for (int l = 1; l < L; l++) {
    MgLevel &D = w->lev[l];
    const size_t plane = (size_t)(D.Z + 2) * D.P;
    D.u = (float *)(mem + off[l]);
    D.f = D.u + plane;
    D.v = D.f + plane;
    D.coef = (const float *)(mem + coff[l]);
    D.cls = (const int *)(mem + ioff[l]);
    D.rw = (const float *)(mem + roff[l]);
  }
  // halos and held nodes start at zero
  e = cudaMemsetAsync(mem + blob.size(), 0, bytes - blob.size(), s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(mem, blob.data(), blob.size(), cudaMemcpyHostToDevice, s);
  char *tmp = nullptr; // the factors
  const size_t lu_bytes = lu.size() * sizeof(double);
  if (e == cudaSuccess && direct) {
    e = dev_malloc(&tmp, lu_bytes);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(tmp, lu.data(), lu_bytes, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k_mg_inverse, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)mg_inverse_smem(MG_MAX_DIRECT, MG_MAX_BAND));
    if (e == cudaSuccess) {
      k_mg_inverse<<<ld / MG_INV_COLS, 32, mg_inverse_smem(cn, band_b), s>>>(cn, band_b, (const double *)tmp,
                                                                                (float *)(mem + o_inv), ld);
      spiffe_note_launches(1);
      e = cudaGetLastError();
    }
  }
  const cudaError_t done = cudaStreamSynchronize(s);
  if (e == cudaSuccess)
    e = done;
  dev_free(tmp);
  if (e != cudaSuccess) {
    s32_mg_free(w);
    return (int)e;
  }

  Mg0 z{};
  z.nz = m->nz;
  z.P = P0;
  z.lo = lo;
  z.hi = hi;
  z.cols = m->nr - 1;
  z.rp = rp0;
  z.nb = nb0;
  const double dz2 = m->dz * m->dz, dr2 = m->dr * m->dr;
  z.a_d = 1 / dz2;
  z.e_d = -2 * (1 / dz2 + 1 / dr2);
  z.e2c_d = z.e_d - 2 / dr2;
  z.a = (float)z.a_d;
  z.e = (float)z.e_d;
  z.e2c = (float)z.e2c_d;
  z.inv_e = (float)(1 / z.e_d);
  z.inv_e2c = (float)(1 / z.e2c_d);
  z.u = (float *)(mem + o_u0);
  z.f = z.u + n0;
  z.crow = (const float *)(mem + o_crow);
  z.drow = (const float *)(mem + o_drow);
  z.cpd = (const double *)(mem + o_cpd);
  z.cmd = (const double *)(mem + o_cmd);
  z.part = (double *)(mem + o_part);
  const MgDense dense{(const float *)(mem + o_inv), (const int *)(mem + o_cidx), cn, ld};
  e = (cudaError_t)mg_graph(w, z, last, fits, direct ? &dense : nullptr, coarse_fits, (float *)(mem + o_scratch),
                            budget * sizeof(float));
  if (e != cudaSuccess) {
    s32_mg_free(w);
    return (int)e;
  }
  w->nlev = L;
  return 0;
}

// the solve on Psi with driving term rhs (null: Laplace), stop rule
// sum|r| < accuracy sum|rhs|, at most max_cycles V-cycles
extern "C" int s32_mg_solve(const DevMesh *m, Mg32Work *w, double *Psi, const double *rhs, const uint8_t *umask,
                            double accuracy, long long max_cycles, PcState *st, long long *iters_out, DevCounts *cnt,
                            cudaStream_t s)
{
  (void)m;
  MgCall c{};
  c.Psi = Psi;
  c.rhs = rhs;
  c.umask = umask;
  c.accuracy = accuracy;
  c.max_cycles = std::min<long long>(max_cycles, 100);
  c.st = st;
  c.iters_out = iters_out;
  c.cnt = cnt;
  k_mg_begin<<<1, 1, 0, s>>>(c, (MgCall *)w->call);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess)
    e = cudaGraphLaunch((cudaGraphExec_t)w->exec, s);
  spiffe_note_launches(2);
  return (int)e;
}
