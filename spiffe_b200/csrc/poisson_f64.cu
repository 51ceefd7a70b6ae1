// spiffe_b200/csrc/poisson_f64.cu -- plain FP64 Poisson correction.
//
// add_poisson_correction (poisson_correction.c:73-454), solve_poisson_cyl
// (poisson.c:17-130) and compute_imposed_Efield (poisson_correction.c:
// 456-562) as device kernels.  The decision whether to solve (the error-
// charge threshold, :258-265) is taken on the device, so a correction needs
// no host round trip.  The red-black SOR runs as one persistent kernel, with
// the mesh in the SMs' shared memory where it fits (k_sor_band; small meshes
// in one cluster's) and over global memory where not (k_sor): each half-sweep
// updates one colour (the reference's colour test, poisson.c:70), every block
// reduces its |residual| sum, and after a barrier all blocks add the per-block
// sums in the same fixed order and take the same stop decision
// (poisson.c:120-121).  Node updates are bit-identical to the reference (a
// colour's nodes read only the other colour); the stop sum is reduced in a
// fixed tree order rather than the reference's serial order, which changes the
// half-sweep count only if the sum lands within rounding distance of the
// threshold.  Built with -fmad=false.
#include "divide.cuh"
#include "modules.cuh"

#include <algorithm>

#include <cooperative_groups.h>

namespace {

constexpr int BX = 32, BY = 8, RT = 256;

// Fixed-order block reduction of one double per thread (blockDim.x*y <= 1024).
__device__ double block_sum(double v, double *sh)
{
  const int t = threadIdx.y * blockDim.x + threadIdx.x, n = blockDim.x * blockDim.y;
  sh[t] = v;
  __syncthreads();
  for (int s = 512; s > 0; s >>= 1) {
    if (t < s && t + s < n)
      sh[t] += sh[t + s];
    __syncthreads();
  }
  const double r = sh[0];
  __syncthreads();
  return r;
}

__device__ bool surface_cell(const DevMesh &m, int16_t fl, int iz, int ir)
{
  return (fl & SPIFFE_FL_IS_METAL) || (iz == 0 && m.left_bc == SPIFFE_NEUMANN) ||
         (iz == m.nz - 1 && m.right_bc == SPIFFE_NEUMANN) || (ir == m.nr - 1 && m.upper_bc == SPIFFE_NEUMANN);
}

// Apparent charge from the flux of E through each cell (:141-182, second pass
// :335-375, where the top-row surface term changes sign).  Per-block partial
// sums of Qsurface and the centroid numerator go to part[2*block+{0,1}].
__global__ void __launch_bounds__(BX *BY) k_apparent_charge(DevMesh m, DevFields<double> f, const double *Az_,
                                                             const double *Ari, const double *Aro, int second,
                                                             double *part)
{
  __shared__ double sh[BX * BY];
  const int ir = blockIdx.x * BX + threadIdx.x, iz = blockIdx.y * BY + threadIdx.y;
  const int nz = m.nz, nr = m.nr, P = m.pitch;
  const double eps = SPIFFE_EPSILON_O;
  double qs = 0, cen = 0;
  if (ir < nr && iz < nz) {
    const size_t i = node(iz, ir, P);
    const double Az = Az_[ir], Ar_inner = Ari[ir], Ar_outer = Aro[ir];
    double dQ;
    if (ir == 0)
      dQ = (f.Er[i + 1] * Ar_outer + (f.Ez[i + P] - f.Ez[i]) * Az) * eps;
    else
      dQ = (f.Er[i + 1] * Ar_outer - f.Er[i] * Ar_inner + (f.Ez[i + P] - f.Ez[i]) * Az) * eps;
    if (surface_cell(m, f.flags[i], iz, ir)) {
      if (iz == 0)
        dQ += f.Ez[i] * Az * eps;
      if (iz == nz - 1)
        dQ -= f.Ez[i + P] * Az * eps;
      if (ir == nr - 1) {
        if (second)
          dQ -= f.Ez[i + 1] * Ar_outer * eps;
        else
          dQ += f.Ez[i + 1] * Ar_outer * eps;
      }
      qs = dQ;
      f.Q[i] = 0;
    } else {
      f.Q[i] = dQ;
      cen = dQ * (iz * m.dz + m.zmin);
    }
  }
  const double s0 = block_sum(qs, sh), s1 = block_sum(cen, sh);
  if (threadIdx.x == 0 && threadIdx.y == 0) {
    const int b = blockIdx.y * gridDim.x + blockIdx.x;
    part[2 * b] = s0;
    part[2 * b + 1] = s1;
  }
}

// Removal of the particles' own charge (:190-242); Qreal partial sums per
// block.  With keys null each share is subtracted by an FP64 atomic, whose
// order varies between runs once three or more particles share a node; with
// keys set, particle ip writes its (node, -share) pairs to entries stride ip,
// ... (unused ones keyed `pad`) for an ordered reduction that applies them in
// particle order, the reference's serial Q[iz][ir] -= ... sequence; shares
// that the mesh's smearing leaves at zero, which change no sum, get no entry.
__global__ void __launch_bounds__(RT) k_remove_charge(DevMesh m, DevFields<double> f, DevBeam64 b,
                                                       const DevCounts *cnt, double *part, int *keys, double *vals,
                                                       long np_bound, int stride, int pad)
{
  __shared__ double sh[RT];
  const long ip = (long)blockIdx.x * RT + threadIdx.x;
  double qreal = 0;
  int at[4] = {0x7fffffff, 0x7fffffff, 0x7fffffff, 0x7fffffff};
  double share[4] = {0, 0, 0, 0};
  if (ip < (long)cnt->np && (b.status[ip] & SPIFFE_PART_ACTIVE)) {
    const long nz = m.nz, nr = m.nr;
    const int P = m.pitch;
    const double dz = m.dz, dr = m.dr;
    const bool lsm = m.modes & SPIFFE_FL_LONGIT_SMEAR, rsm = m.modes & SPIFFE_FL_RADIAL_SMEAR;
    const bool ln = m.left_bc == SPIFFE_NEUMANN, rn = m.right_bc == SPIFFE_NEUMANN, un = m.upper_bc == SPIFFE_NEUMANN;
    const double z = b.z[ip], r = b.r[ip], Q = b.Q[ip];
    const long iz = lsm ? (long)((z - m.zmin) / dz) : (long)((z - m.zmin) / dz + 0.5);
    const long ir = rsm ? (long)(r / dr) : (long)(r / dr + 0.5);
    if (iz >= 0 && iz < nz && ir >= 0 && ir < nr) {
      double fa, fb, fr, fl;
      if (rsm && ir != nr - 1) {
        fa = r / dr - ir;
        fb = 1 - fa;
      } else {
        fb = 1;
        fa = 0;
      }
      if (lsm && iz != nz - 1) {
        fr = (z - m.zmin) / dz - iz;
        fl = 1 - fr;
      } else {
        fl = 1;
        fr = 0;
      }
      const int16_t *F = f.flags;
      const int n0 = node(iz, ir, P), n1 = node(iz + 1, ir, P), n2 = node(iz, ir + 1, P), n3 = node(iz + 1, ir + 1, P);
      if (!((F[n0] & SPIFFE_FL_IS_METAL) || (iz == 0 && ln) || (iz >= nz - 1 && rn) || (ir >= nr - 1 && un))) {
        at[0] = n0;
        share[0] = Q * fb * fl;
        qreal += share[0];
      }
      if (!((F[n1] & SPIFFE_FL_IS_METAL) || (iz == 0 && ln) || (iz >= nz && rn) || (ir >= nr - 1 && un))) {
        at[1] = n1;
        share[1] = Q * fb * fr;
        qreal += share[1];
      }
      if (!((F[n2] & SPIFFE_FL_IS_METAL) || (iz == 0 && ln) || (iz >= nz - 1 && rn) || (ir >= nr && un))) {
        at[2] = n2;
        share[2] = Q * fa * fl;
        qreal += share[2];
      }
      if (!((F[n3] & SPIFFE_FL_IS_METAL) || (iz == 0 && ln) || (iz >= nz && rn) || (ir >= nr && un))) {
        at[3] = n3;
        share[3] = Q * fa * fr;
        qreal += share[3];
      }
    }
  }
  if (keys) {
    if (ip < np_bound) {
      const bool lsm = m.modes & SPIFFE_FL_LONGIT_SMEAR, rsm = m.modes & SPIFFE_FL_RADIAL_SMEAR;
      int e = 0;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        if (((k & 1) && !lsm) || ((k & 2) && !rsm))
          continue;
        keys[stride * ip + e] = at[k] == 0x7fffffff ? pad : at[k];
        vals[stride * ip + e] = at[k] == 0x7fffffff ? 0.0 : -share[k];
        e++;
      }
    }
  } else {
    // (without smearing three of the four shares are 0 and change nothing;
    // adding them took 164 of the kernel's 223 us a million particles)
    for (int k = 0; k < 4; k++)
      if (share[k] != 0)
        atomicAdd(f.Q + at[k], -share[k]);
  }
  const double s = block_sum(qreal, sh);
  if (threadIdx.x == 0)
    part[blockIdx.x] = s;
}

// Sum over a (rows x cols) window of a pitched array, |x| when absval.
__global__ void __launch_bounds__(BX *BY) k_region_sum(const double *a, int rows, int cols, int P, int absval,
                                                        double *part)
{
  __shared__ double sh[BX * BY];
  const int ir = blockIdx.x * BX + threadIdx.x, iz = blockIdx.y * BY + threadIdx.y;
  double v = 0;
  if (ir < cols && iz < rows) {
    v = a[node(iz, ir, P)];
    if (absval)
      v = fabs(v);
  }
  const double s = block_sum(v, sh);
  if (threadIdx.x == 0 && threadIdx.y == 0)
    part[blockIdx.y * gridDim.x + blockIdx.x] = s;
}

// Serial fixed-order sum of n partials (strided by `stride`) into *out.
__global__ void k_finish_sum(const double *part, int n, int stride, double *out)
{
  __shared__ double sh[1024];
  double v = 0;
  for (int i = threadIdx.x; i < n; i += blockDim.x)
    v += part[(size_t)i * stride];
  sh[threadIdx.x] = v;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s)
      sh[threadIdx.x] += sh[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0)
    *out = sh[0];
}

// error-charge threshold test (:258-265).  The reference sums Qerror
// serially, iz outer and ir inner (:245-248); the device's tree sum of the
// same values differs from it by at most 2 gamma_(n-1) sum|Q| (n terms,
// gamma_k = k u / (1 - k u), u = 2^-53).  When |Qerror| is farther than that
// from a positive threshold the decision is the reference's; otherwise (an
// error charge at the level of rounding noise, as with no particles left)
// this thread redoes the sum in the reference's order.
__global__ void k_pc_decide(PcState *st, double threshold, const double *Q, int nz, int nr, int P,
                            const double *abs_sum)
{
  if (threshold > 0 && abs_sum) {
    const double n = (double)nz * (double)nr, u = 1.1102230246251565e-16;
    const double margin = 2.0 * (n * u / (1.0 - n * u)) * *abs_sum * 1.0001 + 1e-300;
    if (fabs(fabs(st->Qerror) - threshold) <= margin) {
      double q = 0;
      for (int iz = 0; iz < nz; iz++)
        for (int ir = 0; ir < nr; ir++)
          q += Q[node(iz, ir, P)];
      st->Qerror = q;
    }
  }
  const double Qerror = st->Qerror, Qreal = st->Qreal;
  int skip = (threshold > 0 && fabs(Qerror) < threshold) ||
             (threshold < 0 && (Qreal == 0 || fabs(Qerror / Qreal) < fabs(threshold)));
  st->do_solve = !skip;
}

// Q -> -Q/(V eps0) over iz < nz, ir < nr (:268-274)
__global__ void __launch_bounds__(BX *BY) k_scale_rhs(DevMesh m, DevFields<double> f, const double *volume,
                                                       const PcState *st)
{
  if (!st->do_solve)
    return;
  const int ir = blockIdx.x * BX + threadIdx.x, iz = blockIdx.y * BY + threadIdx.y;
  if (ir < m.nr && iz < m.nz) {
    const size_t i = node(iz, ir, m.pitch);
    f.Q[i] = -f.Q[i] / (volume[ir] * SPIFFE_EPSILON_O);
  }
}

// poisson_guess (:564-615)
__global__ void __launch_bounds__(BX *BY) k_guess(DevMesh m, DevFields<double> f, int code, const PcState *st)
{
  if (!st->do_solve)
    return;
  const int ir = blockIdx.x * BX + threadIdx.x, iz = blockIdx.y * BY + threadIdx.y;
  if (ir >= m.nr || iz >= m.nz)
    return;
  const size_t i = node(iz, ir, m.pitch);
  const double charge = st->Qerror;
  if (code == 1)
    f.Psi[i] = charge / (SPIFFE_PIx2 * SPIFFE_EPSILON_O) * log((ir ? ir : 0.5) * m.dr);
  else if (code == 2) {
    const double zz = (iz * m.dz + m.zmin) - st->centroid, rr = m.dr * (ir + 0.5);
    const double dist = sqrt(zz * zz + rr * rr);
    f.Psi[i] = charge / (4 * SPIFFE_PI * SPIFFE_EPSILON_O * dist);
  } else if (code == 3)
    f.Psi[i] = 0;
}

// Bounded grid barrier for a cooperative launch: returns false (and raises
// the device error bit) if the other blocks do not arrive within `limit` polls.
__device__ bool grid_barrier(unsigned *count, unsigned *gen, unsigned nblocks, DevCounts *cnt)
{
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0 && threadIdx.y == 0) {
    ok = 1;
    volatile unsigned *vgen = gen;
    const unsigned g = *vgen;
    __threadfence();
    if (atomicAdd(count, 1u) == nblocks - 1) {
      atomicExch(count, 0u);
      __threadfence();
      atomicAdd(gen, 1u);
    } else {
      unsigned long long polls = 0;
      while (*vgen == g) {
        if (++polls > (1ull << 26)) {
          ok = 0;
          atomicOr(&cnt->error, SPIFFE_DEV_ERR_BARRIER);
          break;
        }
        __nanosleep(64);
      }
    }
    __threadfence();
  }
  __syncthreads();
  return ok;
}

struct SorArgs {
  double *Psi;
  const double *rhs; // null for the Laplace solve of the imposed potential
  const int16_t *flags;
  const double *omega;       // omega[n] for half-sweep n
  const double *crow, *drow; // c and d of each row ir >= 1 (poisson.c:357-358)
  double a, e, c4_axis, e2c_axis, accuracy; // 4c and e-2c of the axis row (poisson.c:361, :386-387)
  const double *driving;     // sum |rhs|
  long long limit;
  double *partials; // 2*gridDim.x doubles
  unsigned *bar_count, *bar_gen;
  PcState *st; // iterations and final residual; do_solve gate (may be null)
  long long *iterations_out;
};

// solve_poisson_cyl (poisson.c:17-130): rows ir = 0..nr-2 of the iz the
// boundary conditions leave free; half-sweep n updates the nodes with
// (ir+iz)%2 == n%2.  Each block owns whole iz rows (block-strided) and its
// threads visit only that row's nodes of the current colour, so a warp reads
// every other Psi of a row.  Psi of neighbouring rows was written by other
// blocks in the previous half-sweep, so it is read through L2 (ld.cg).
__global__ void __launch_bounds__(RT) k_sor(DevMesh m, SorArgs s, DevCounts *cnt)
{
  __shared__ double sh[RT];
  if (s.st && !s.st->do_solve)
    return;
  const int nz = m.nz, nr = m.nr, P = m.pitch;
  const int lo = m.left_bc == SPIFFE_DIRICHLET ? 0 : 1, hi = m.right_bc == SPIFFE_DIRICHLET ? nz - 1 : nz - 2;
  const int cols = nr - 1, rows = hi - lo + 1;
  const double a = s.a, e = s.e;
  const double thr = s.accuracy * *s.driving;
  long long result = -1;
  double total = 0;
  for (long long n = 0; n < s.limit; n++) {
    const double omega = s.omega[n];
    const int colour = (int)(n & 1);
    double acc = 0;
    for (int row = blockIdx.x; row < rows; row += gridDim.x) {
      const int iz = lo + row;
      const int parity = (colour + iz) & 1; // ir with (ir+iz)%2 == colour
      const size_t base = node(iz, 0, P);
      // the left and right Dirichlet rows mirror their only neighbour (poisson.c:369-375, :404-410)
      const long up = (iz == 0 && lo == 0) ? P : (iz == nz - 1 && hi == nz - 1 ? -P : P);
      const long dn = (iz == 0 && lo == 0) ? P : -P;
      for (int ir = 2 * threadIdx.x + parity; ir < cols; ir += 2 * RT) {
        const size_t i = base + ir;
        if (s.flags[i] & SPIFFE_FL_IS_METAL)
          continue;
        const double left = __ldcg(s.Psi + i + up), right = __ldcg(s.Psi + i + dn);
        const double drive = s.rhs ? s.rhs[i] : 0;
        const double self = __ldcg(s.Psi + i);
        double residual;
        if (ir == 0) {
          residual = a * (left + right) + s.c4_axis * __ldcg(s.Psi + i + 1) + s.e2c_axis * self - drive;
          __stcg(s.Psi + i, self - omega * residual / s.e2c_axis);
        } else {
          residual = a * (left + right) + s.crow[ir] * __ldcg(s.Psi + i + 1) + s.drow[ir] * __ldcg(s.Psi + i - 1) +
                     e * self - drive;
          __stcg(s.Psi + i, self - omega * residual / e);
        }
        acc += fabs(residual);
      }
    }
    // partial sums alternate between two halves of the buffer, so a block
    // that runs ahead cannot overwrite sums another block is still reading
    double *part = s.partials + (size_t)(n & 1) * gridDim.x;
    const double bs = block_sum(acc, sh);
    if (threadIdx.x == 0)
      __stcg(part + blockIdx.x, bs);
    __threadfence();
    if (!grid_barrier(s.bar_count, s.bar_gen, gridDim.x, cnt))
      return;
    // every block forms the same fixed-order sum of the partials
    double v = 0;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += RT)
      v += __ldcg(part + b);
    total = block_sum(v, sh);
    if (n > 0 && (total < thr || total == 0)) {
      result = n;
      break;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (s.iterations_out)
      *s.iterations_out = result;
    if (s.st) {
      s.st->iterations = result;
      s.st->residual = total;
    }
    cnt->sor_halfsweeps += result >= 0 ? result + 1 : s.limit;
    cnt->sor_solves += 1;
  }
}

// ---- the same SOR with its rows in shared memory
//
// k_sor reads Psi through L2 and a half-sweep of it costs 16.9 us on the
// 3001 x 821 gun (4.7 us on a mesh a hundredth its size): the barrier of 592
// blocks and the L2 latencies between two of them.  Here each SM holds a band
// of rows of Psi in shared memory for the whole solve, one CTA an SM, and
// half a row crosses to each neighbour after a half-sweep.  A row lies as its
// even columns and then its odd ones, so that the nodes of one colour are
// consecutive; the driving term is kept in that order too (rs), and a
// half-sweep's part of it is loaded while the CTA waits at the barrier.  The
// arithmetic of a node is k_sor's, operation by operation, the division by
// the constant diagonal with a product and four fused corrections
// (div_const), so Psi has the same bits; the stop sum is again formed in one
// fixed order by every CTA.  Measured a half-sweep (B200; random charge / a
// bunch's): 3001 x 821 8.3 / 10.1 us, 1501 x 1001 5.9 / 7.0, 1201 x 329 (8.5
// before) 3.9 / 4.3, 301 x 83 3.2: about 3 of it the barrier with the sums
// and the exchange, the rest instruction issue (FP64 without contraction).
// 1024 threads spilled their prefetched driving terms (8.7 / 12.8), 512 had
// too few warps (11.7 / 17.9), a barrier of one tagged word a band in place of
// the counter cost 3 us more.
constexpr int SB_NT = 768;     // threads of a CTA
constexpr int SB_CLUSTER = 16; // blocks of the cluster form, at most

struct SorBand {
  int R, H;           // rows of a band; half-row length (doubles)
  double inv_e, inv_e2c;
  double *rs;         // driving term [rows][2][H]
  double *xb;         // [2][G][2][H]: updated halves of the bands' first and last rows
  unsigned long long *bar; // [0] arrivals, [16] abort
};

// RK: rows of a band that a thread takes, at most.  CLUSTER: the grid is one
// thread-block cluster, whose barrier takes the place of the counter in
// global memory; the bands write their edge rows and sums straight into the
// others' shared memory, so that nothing is fetched behind the barrier.  301 x
// 83: 3.6 -> 2.1 us a half-sweep, of which the barriers are still more than half.
template <int RK, bool CLUSTER>
__global__ void __launch_bounds__(SB_NT, 1) k_sor_band(DevMesh m, SorArgs s, SorBand sb, DevCounts *cnt)
{
  extern __shared__ double2 sb_smem[];
  __shared__ double sh[SB_NT / 32];
  __shared__ double total_sh;
  __shared__ double part_sh[2][SB_CLUSTER]; // CLUSTER: every band's sum, by colour
  __shared__ int ok_sh;
  if (s.st && !s.st->do_solve)
    return;
  namespace cg = cooperative_groups;
  double *S = reinterpret_cast<double *>(sb_smem);
  const int nz = m.nz, nr = m.nr, P = m.pitch, H = sb.H, G = gridDim.x, b = blockIdx.x, tid = threadIdx.x;
  const int lo = m.left_bc == SPIFFE_DIRICHLET ? 0 : 1, hi = m.right_bc == SPIFFE_DIRICHLET ? nz - 1 : nz - 2;
  const int cols = nr - 1, first = lo + b * sb.R, nrow = min(sb.R, hi + 1 - first);
  double *C = S + (size_t)(sb.R + 2) * 2 * H, *D = C + 2 * H; // c and d of each column, in a row's order
  // this thread's columns: nodes j, j+1 of each half row, in rows g, g+groups, ...
  const int W = ((((cols + 1) >> 1) + 1) / 2 + 31) & ~31, groups = SB_NT / W, g = tid / W, j = 2 * (tid - g * W);
  const bool on = g < groups && 2 * j < cols;
  // rows first-1 .. first+nrow of Psi and the band's rows of the driving term
  for (int k = tid; k < (nrow + 2) * (nr + 1); k += SB_NT) {
    const int r = k / (nr + 1), ir = k - r * (nr + 1), iz = first - 1 + r;
    S[(size_t)r * 2 * H + (ir & 1) * H + (ir >> 1)] = iz >= 0 && iz <= nz ? s.Psi[node(iz, ir, P)] : 0.0;
  }
  for (int ir = tid; ir < 2 * H; ir += SB_NT) {
    const bool in = ir < cols;
    C[(ir & 1) * H + (ir >> 1)] = in ? (ir ? s.crow[ir] : s.c4_axis) : 0.0;
    D[(ir & 1) * H + (ir >> 1)] = in && ir ? s.drow[ir] : 0.0;
  }
  double *rs = sb.rs + (size_t)b * sb.R * 2 * H;
  for (int k = tid; k < nrow * cols; k += SB_NT) {
    const int r = k / cols, ir = k - r * cols;
    rs[(size_t)r * 2 * H + (ir & 1) * H + (ir >> 1)] = s.rhs ? s.rhs[node(first + r, ir, P)] : 0.0;
  }
  // which of the thread's nodes are updated: bits 4k + 2 half + q
  unsigned upd = 0;
  if (on)
    for (int k = 0; k < RK; k++)
      for (int t = 0; t < 4; t++) {
        const int ir = 2 * (j + (t & 1)) + (t >> 1), r = g + k * groups;
        if (ir < cols && r < nrow && !(s.flags[node(first + r, ir, P)] & SPIFFE_FL_IS_METAL))
          upd |= 1u << (4 * k + t);
      }
  const double a = s.a, e = s.e, y = sb.inv_e, thr = s.accuracy * *s.driving;
  double2 rh[RK]; // the coming half-sweep's driving terms
  auto load_rh = [&](int colour) {
#pragma unroll
    for (int k = 0; k < RK; k++) {
      const int r = g + k * groups;
      if (on && r < nrow)
        rh[k] = __ldcg(reinterpret_cast<const double2 *>(rs + (size_t)r * 2 * H + ((colour + first + r) & 1) * H + j));
    }
  };
  if (CLUSTER)
    cg::this_cluster().sync(); // every band has its rows before a neighbour writes to them
  else
    __syncthreads();
  load_rh(0);
  long long result = -1;
  double total = 0;
  for (long long n = 0; n < s.limit; n++) {
    const double omega = __ldg(s.omega + n);
    const int colour = (int)(n & 1);
    double acc = 0;
    if (on)
#pragma unroll
      for (int k = 0; k < RK; k++) {
        const int r = g + k * groups;
        if (r < nrow) {
          const int iz = first + r, h = (colour + iz) & 1; // the colour's columns have parity h
          double *row = S + (size_t)(r + 1) * 2 * H, *x = row + h * H + j;
          // the left and right Dirichlet rows mirror their only neighbour (poisson.c:369-375, :404-410)
          const double *up = (iz == nz - 1 && hi == nz - 1) ? x - 2 * H : x + 2 * H;
          const double *dn = (iz == 0 && lo == 0) ? x + 2 * H : x - 2 * H;
          const double2 l = *reinterpret_cast<const double2 *>(up), q = *reinterpret_cast<const double2 *>(dn);
          const double2 o = *reinterpret_cast<const double2 *>(row + (1 - h) * H + j);
          const double2 c = *reinterpret_cast<const double2 *>(C + h * H + j), d = *reinterpret_cast<const double2 *>(D + h * H + j);
          double2 v = *reinterpret_cast<const double2 *>(x);
          const unsigned bits = upd >> (4 * k + 2 * h);
          double rx, ry, ex = e, yx = y;
          if (h) { // (the same for the whole warp)
            rx = a * (l.x + q.x) + c.x * o.y + d.x * o.x + e * v.x - rh[k].x;
            ry = a * (l.y + q.y) + c.y * row[j + 2] + d.y * o.y + e * v.y - rh[k].y;
          } else {
            if (j == 0) { // the axis, whose d is 0
              ex = s.e2c_axis;
              yx = sb.inv_e2c;
            }
            rx = a * (l.x + q.x) + c.x * o.x + d.x * (j ? row[H + j - 1] : 0.0) + ex * v.x - rh[k].x;
            ry = a * (l.y + q.y) + c.y * o.y + d.y * o.x + e * v.y - rh[k].y;
          }
          const double tx = omega * rx, ty = omega * ry;
          double qx = div_const(tx, ex, yx), qy = div_const(ty, e, y);
          if (div_rare(tx) || div_rare(ty)) {
            if (div_rare(tx))
              qx = div_scaled(tx, ex, yx);
            if (div_rare(ty))
              qy = div_scaled(ty, e, y);
          }
          if (bits & 1u) {
            v.x -= qx;
            acc += fabs(rx);
          }
          if (bits & 2u) {
            v.y -= qy;
            acc += fabs(ry);
          }
          *reinterpret_cast<double2 *>(x) = v;
          if (CLUSTER) {
            // into the neighbours' halo rows: they read this colour's half of
            // them in the next half-sweep, behind the barrier
            if (r == 0 && b > 0)
              *reinterpret_cast<double2 *>(cg::this_cluster().map_shared_rank(S, b - 1) + (size_t)(sb.R + 1) * 2 * H + h * H + j) = v;
            if (r == nrow - 1 && b < G - 1)
              *reinterpret_cast<double2 *>(cg::this_cluster().map_shared_rank(S, b + 1) + h * H + j) = v;
          } else {
            double *xo = sb.xb + ((size_t)colour * G + b) * 2 * H + j;
            if (r == 0)
              __stcg(reinterpret_cast<double2 *>(xo), v);
            if (r == nrow - 1)
              __stcg(reinterpret_cast<double2 *>(xo + H), v);
          }
        }
      }
    // the next half-sweep's driving terms arrive while the CTA waits
    load_rh(1 - colour);
    for (int o = 16; o > 0; o >>= 1)
      acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((tid & 31) == 0)
      sh[tid >> 5] = acc;
    __syncthreads();
    // the sums alternate between two halves of the buffer, so a CTA that runs
    // ahead cannot overwrite sums another is still reading
    double *part = s.partials + (size_t)colour * G;
    if (tid < 32) {
      double v = tid < SB_NT / 32 ? sh[tid] : 0.0;
      for (int o = 16; o > 0; o >>= 1)
        v += __shfl_down_sync(0xffffffffu, v, o);
      if (CLUSTER) {
        v = __shfl_sync(0xffffffffu, v, 0);
        if (tid < G)
          cg::this_cluster().map_shared_rank(&part_sh[0][0], tid)[colour * SB_CLUSTER + b] = v;
      } else if (tid == 0) {
        __stcg(part + b, v);
        int ok = 1;
        asm volatile("fence.acq_rel.gpu;" ::: "memory");
        asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(sb.bar), "l"(1ull) : "memory");
        const unsigned long long target = (unsigned long long)G * (unsigned long long)(n + 1);
        unsigned long long polls = 0, seen = 0, gone = 0;
        for (;;) {
          asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(seen) : "l"(sb.bar) : "memory");
          if (seen >= target)
            break;
          if ((++polls & 63) == 0) // bounded: 2^24 polls, or another band has given up
            asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(gone) : "l"(sb.bar + 16) : "memory");
          if (gone || polls > (1ull << 24)) {
            if (!gone) {
              atomicOr(&cnt->error, SPIFFE_DEV_ERR_BARRIER);
              asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(sb.bar + 16), "l"(1ull) : "memory");
            }
            ok = 0;
            break;
          }
        }
        ok_sh = ok;
      }
    }
    if (CLUSTER) {
      cg::this_cluster().sync();
      // every warp forms the same sum of the partials
      double v = (tid & 31) < G ? part_sh[colour][tid & 31] : 0.0;
      for (int o = 16; o > 0; o >>= 1)
        v += __shfl_down_sync(0xffffffffu, v, o);
      total = __shfl_sync(0xffffffffu, v, 0);
    } else {
      __syncthreads();
      if (!ok_sh)
        return;
      if (tid >= SB_NT - 32) { // the last warp: every CTA forms the same sum of the partials
        double v = 0;
        for (int k = tid - (SB_NT - 32); k < G; k += 32)
          v += __ldcg(part + k);
        for (int o = 16; o > 0; o >>= 1)
          v += __shfl_down_sync(0xffffffffu, v, o);
        if (tid == SB_NT - 32)
          total_sh = v;
      } else { // the others: the neighbours' rows
        const double *xi = sb.xb + (size_t)colour * G * 2 * H;
        for (int k = 2 * tid; k < 2 * H; k += 2 * (SB_NT - 32)) {
          const bool above = k >= H;
          const int t = above ? k - H : k, nb = above ? b + 1 : b - 1, iz = above ? first + nrow : first - 1;
          if (nb < 0 || nb >= G)
            continue;
          const double2 v = __ldcg(reinterpret_cast<const double2 *>(xi + (size_t)nb * 2 * H + (above ? 0 : H) + t));
          *reinterpret_cast<double2 *>(S + (size_t)(above ? nrow + 1 : 0) * 2 * H + ((colour + iz) & 1) * H + t) = v;
        }
      }
      __syncthreads();
      total = total_sh;
    }
    if (n > 0 && (total < thr || total == 0)) {
      result = n;
      break;
    }
  }
  for (int k = tid; k < nrow * cols; k += SB_NT) {
    const int r = k / cols, ir = k - r * cols;
    s.Psi[node(first + r, ir, P)] = S[(size_t)(r + 1) * 2 * H + (ir & 1) * H + (ir >> 1)];
  }
  if (b == 0 && tid == 0) {
    if (s.iterations_out)
      *s.iterations_out = result;
    if (s.st) {
      s.st->iterations = result;
      s.st->residual = total;
    }
    cnt->sor_halfsweeps += result >= 0 ? result + 1 : s.limit;
    cnt->sor_solves += 1;
  }
}

// rows of a thread for bands of R rows (0: the mesh's rows are too wide)
int sb_rows(int cols, int R)
{
  const int W = ((((cols + 1) >> 1) + 1) / 2 + 31) & ~31, groups = SB_NT / W;
  return groups ? (R + groups - 1) / groups : 0;
}

// An instance holds the driving terms of all a thread's rows in registers, so one
// with rows to spare spills more: 36 bytes a thread with seven, 68 with eight, none
// with four (3001 x 821, seven rows a thread: 8.3 us a half-sweep, 8.5 with the
// instance for eight; 2400 x 900, seven: 7.6 and 7.9).  Five and six take seven's.
const void *sb_kernel(int rows)
{
  return rows <= 2   ? (const void *)k_sor_band<2, false>
         : rows <= 4 ? (const void *)k_sor_band<4, false>
         : rows <= 7 ? (const void *)k_sor_band<7, false>
         : rows <= 8 ? (const void *)k_sor_band<8, false>
                     : nullptr;
}

// The cluster form's bands: a power of two of blocks, each with rows, of at
// most SB_CLUSTER_ROWS rows a thread; 0 where there is none.  With two rows a
// thread the sixteen SMs are faster than all with a barrier through L2 (601 x
// 83: 2.8 against 3.75 us a half-sweep, 201 x 300: 2.7 against 3.35), with
// three and four no longer (801 x 100: 3.4 against 3.4, 601 x 165: 4.1 against 3.9).
constexpr int SB_CLUSTER_ROWS = 2;
int sb_cluster(int rows, int cols, int &R)
{
  for (int G = SB_CLUSTER; G > 1; G /= 2) {
    R = (rows + G - 1) / G;
    const int per_thread = sb_rows(cols, R);
    if (per_thread > SB_CLUSTER_ROWS || !per_thread)
      return 0; // fewer blocks would have more rows
    if ((rows + R - 1) / R == G)
      return G;
  }
  return 0;
}

cudaLaunchConfig_t sb_cluster_config(int G, size_t smem, cudaStream_t s, cudaLaunchAttribute *at)
{
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = (unsigned)G;
  at->val.clusterDim.y = at->val.clusterDim.z = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = dim3(G);
  c.blockDim = dim3(SB_NT);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = at;
  c.numAttrs = 1;
  return c;
}

// Ez, Er -= grad Psi (:288-326) with the FDTD boundary copies; one writer per node.
__global__ void __launch_bounds__(BX *BY) k_subtract_gradient(DevMesh m, DevFields<double> f, const PcState *st)
{
  if (!st->do_solve)
    return;
  const int ir = blockIdx.x * BX + threadIdx.x, iz = blockIdx.y * BY + threadIdx.y;
  const int nz = m.nz, nr = m.nr, P = m.pitch;
  if (ir > nr || iz > nz)
    return;
  const size_t i = node(iz, ir, P);
  const bool leftN = m.left_bc == SPIFFE_NEUMANN, rightN = m.right_bc == SPIFFE_NEUMANN;
  if (ir < nr && iz >= 1 && iz <= nz - 1) {
    double v = f.Ez[i];
    if (!(f.flags[i] & SPIFFE_FL_EZ_ZERO))
      v -= -(f.Psi[i] - f.Psi[i - P]) / m.dz;
    if (ir == nr - 1)
      v = 0.0;
    f.Ez[i] = v;
    if (iz == 1)
      f.Ez[node(0, ir, P)] = ir == nr - 1 ? 0.0 : (leftN ? v : -v);
    if (iz == nz - 1)
      f.Ez[node(nz, ir, P)] = ir == nr - 1 ? 0.0 : (rightN ? v : -v);
  }
  if (iz <= nz - 1) {
    const bool zero_row = (leftN && iz == 0) || (rightN && iz == nz - 1);
    if (ir >= 1) {
      double v = f.Er[i];
      if (!(f.flags[i] & SPIFFE_FL_ER_ZERO))
        v -= -(f.Psi[i] - f.Psi[i - 1]) / m.dr;
      f.Er[i] = zero_row ? 0.0 : v;
      if (ir == 1)
        f.Er[node(iz, 0, P)] = zero_row ? 0.0 : -v;
    }
  }
}

// EzImposed, ErImposed = -factor grad PsiImposed (:523-561).
__global__ void __launch_bounds__(BX *BY) k_imposed_field(DevMesh m, DevFields<double> f, double ff)
{
  const int ir = blockIdx.x * BX + threadIdx.x, iz = blockIdx.y * BY + threadIdx.y;
  const int nz = m.nz, nr = m.nr, P = m.pitch;
  if (ir > nr || iz > nz)
    return;
  const size_t i = node(iz, ir, P);
  const bool leftN = m.left_bc == SPIFFE_NEUMANN, rightN = m.right_bc == SPIFFE_NEUMANN;
  if (ir < nr && iz >= 1 && iz <= nz - 1) {
    double v = f.EzImposed[i];
    if (!(f.flags[i] & SPIFFE_FL_EZ_ZERO))
      v = -ff * (f.PsiImposed[i] - f.PsiImposed[i - P]) / m.dz;
    if (ir == nr - 1)
      v = 0.0;
    f.EzImposed[i] = v;
    if (iz == 1)
      f.EzImposed[node(0, ir, P)] = ir == nr - 1 ? 0.0 : (leftN ? v : -v);
    if (iz == nz - 1)
      f.EzImposed[node(nz, ir, P)] = ir == nr - 1 ? 0.0 : (rightN ? v : -v);
  }
  if (iz <= nz - 1) {
    const bool zero_row = (leftN && iz == 0) || (rightN && iz == nz - 1);
    if (ir >= 1) {
      double v = f.ErImposed[i];
      if (!(f.flags[i] & SPIFFE_FL_ER_ZERO))
        v = -ff * (f.PsiImposed[i] - f.PsiImposed[i - 1]) / m.dr;
      f.ErImposed[i] = zero_row ? 0.0 : v;
      if (ir == 1)
        f.ErImposed[node(iz, 0, P)] = zero_row ? 0.0 : -v;
    }
  }
}

__global__ void k_set_state(PcState *st, double *qs_cen, double *qreal, double *qerr, int space_charge)
{
  st->Qsurface = qs_cen[0];
  st->centroid = qs_cen[1];
  st->Qreal = space_charge ? *qreal : 0.0;
  st->Qerror = *qerr;
}

} // namespace

// ---------------------------------------------------------------- host side


extern "C" int spiffe_poisson64_setup(const DevMesh *m, Poisson64Work *w, long long np_capacity, cudaStream_t s)
{
  const int nr = m->nr, nz = m->nz;
  const double dr = m->dr, dz = m->dz, dr2 = dr * dr, drdz = dr * dz;
  double *Az = new double[nr + 1], *Ari = new double[nr + 1], *Aro = new double[nr + 1], *vol = new double[nr + 1];
  for (int ir = 0; ir <= nr; ir++) {
    if (ir == 0) {
      Ari[ir] = Aro[ir] = SPIFFE_PI * drdz;
      Az[ir] = dr2 / 4 * SPIFFE_PI;
    } else {
      Ari[ir] = SPIFFE_PI * (2 * ir - 1) * drdz;
      Aro[ir] = SPIFFE_PI * (2 * ir + 1) * drdz;
      Az[ir] = SPIFFE_PI * dr2 / 4 * (double)((long)(2 * ir + 1) * (2 * ir + 1) - (long)(2 * ir - 1) * (2 * ir - 1));
    }
    vol[ir] = Az[ir] * dz;
  }
  cudaError_t e = cudaSuccess;
  const size_t gx = (nr + 1 + BX - 1) / BX, gy = (nz + 1 + BY - 1) / BY;
  size_t parts = 2 * gx * gy;
  const size_t pblocks = (size_t)blocks_for(np_capacity > 0 ? np_capacity : 1, RT);
  if (pblocks > parts)
    parts = pblocks;
  if (parts < 4096)
    parts = 4096;
  if (!w->Az) {
    DeviceSlab d;
    d.add(&w->Az, nr + 1);
    d.add(&w->Ari, nr + 1);
    d.add(&w->Aro, nr + 1);
    d.add(&w->volume, nr + 1);
    d.add(&w->crow, nr + 1);
    d.add(&w->drow, nr + 1);
    d.add(&w->scalars, 8);
    d.add(&w->bar, 2);
    d.add(&w->st, 1);
    d.add(&w->iters, 1);
    e = d.make();
    if (e == cudaSuccess) e = cudaMemsetAsync(w->bar, 0, sizeof(unsigned) * 2, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(w->st, 0, sizeof(PcState), s);
  }
  if (e == cudaSuccess && w->part_n < parts) {
    dev_free(w->part);
    e = dev_malloc(&w->part, sizeof(double) * parts);
    w->part_n = e == cudaSuccess ? parts : 0;
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(w->Az, Az, sizeof(double) * (nr + 1), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(w->Ari, Ari, sizeof(double) * (nr + 1), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(w->Aro, Aro, sizeof(double) * (nr + 1), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(w->volume, vol, sizeof(double) * (nr + 1), cudaMemcpyHostToDevice, s);
  // SOR row coefficients with the reference's expressions (poisson.c:355-361)
  double *crow = new double[nr + 1], *drow = new double[nr + 1];
  for (int ir = 0; ir <= nr; ir++) {
    if (ir != 0) {
      crow[ir] = 1 / (dr * dr) * (1 + 1. / (2 * ir));
      drow[ir] = 1 / (dr * dr) * (1 - 1. / (2 * ir));
    } else
      crow[ir] = drow[ir] = 1 / (dr * dr);
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(w->crow, crow, sizeof(double) * (nr + 1), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(w->drow, drow, sizeof(double) * (nr + 1), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  delete[] crow;
  delete[] drow;
  delete[] Az;
  delete[] Ari;
  delete[] Aro;
  delete[] vol;
  if (e == cudaSuccess && !w->sor_grid) {
    int dev = 0, sms = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_sor, RT, 0);
    if (per > 4)
      per = 4;
    w->sor_grid = sms * (per > 0 ? per : 1);
    if ((size_t)(2 * w->sor_grid) > w->part_n)
      w->sor_grid = (int)(w->part_n / 2);
    // bands in shared memory, where the mesh fits the SMs' and its rows a
    // CTA's threads: about 4 million nodes (fewer of very long rows); beyond
    // that k_sor, which has no such limit
    int max_smem = 0;
    cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    const int lo = m->left_bc == SPIFFE_DIRICHLET ? 0 : 1, hi = m->right_bc == SPIFFE_DIRICHLET ? nz - 1 : nz - 2;
    const int rows = hi - lo + 1, H = ((nr + 2) / 2 + 1) / 2 * 2;
    int G = std::max(1, std::min(sms, rows / 2)), R = (rows + G - 1) / G, per_thread = sb_rows(nr - 1, R);
    const void *k = per_thread ? sb_kernel(per_thread) : nullptr;
    auto bytes = [&](int r) { return (size_t)(r + 4) * 2 * H * sizeof(double); };
    cudaFuncAttributes fa{};
    int Rc = 0;
    const int Gc = sb_cluster(rows, nr - 1, Rc);
    if (Gc) {
      const void *kc = (const void *)k_sor_band<SB_CLUSTER_ROWS, true>;
      cudaLaunchAttribute at{};
      const cudaLaunchConfig_t c = sb_cluster_config(Gc, bytes(Rc), s, &at);
      int fits = 0;
      if (cudaFuncGetAttributes(&fa, kc) == cudaSuccess && bytes(Rc) + fa.sharedSizeBytes <= (size_t)max_smem &&
          cudaFuncSetAttribute(kc, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem - (int)fa.sharedSizeBytes) == cudaSuccess &&
          cudaFuncSetAttribute(kc, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
          cudaOccupancyMaxActiveClusters(&fits, kc, &c) == cudaSuccess && fits > 0) {
        k = kc;
        R = Rc;
        w->band_cluster = Gc;
      }
      cudaGetLastError();
    }
    const size_t smem = bytes(R);
    if (e == cudaSuccess && k && cudaFuncGetAttributes(&fa, k) == cudaSuccess && smem + fa.sharedSizeBytes <= (size_t)max_smem) {
      e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem - (int)fa.sharedSizeBytes);
      const int used = (rows + R - 1) / R;
      const size_t rs = (size_t)rows * 2 * H, xb = (size_t)4 * used * H;
      if (e == cudaSuccess) e = dev_malloc(&w->band_mem, (rs + xb) * sizeof(double) + 32 * sizeof(unsigned long long));
      if (e == cudaSuccess) {
        w->band_kernel = k;
        w->band_grid = used;
        w->band_R = R;
        w->band_H = H;
        w->band_lo = lo;
        w->band_hi = hi;
        w->band_smem = smem;
        w->band_xb = w->band_mem + rs;
        w->band_bar = (unsigned long long *)(w->band_xb + xb);
      }
    }
  }
  return (int)e;
}

extern "C" void spiffe_poisson64_free(Poisson64Work *w)
{
  dev_free(w->Az); // with the others
  dev_free(w->part);
  dev_free(w->omega);
  dev_free(w->band_mem);
  *w = Poisson64Work();
}

// Chebyshev over-relaxation sequence, poisson.c:342-344, :416-419.
static int ensure_omega(const DevMesh *m, Poisson64Work *w, long long limit, cudaStream_t s)
{
  if (w->omega && w->omega_n >= limit)
    return 0;
  dev_free(w->omega);
  const double rz = m->dz / m->dr;
  const double rj = (cos(SPIFFE_PI / m->nz) + rz * rz * cos(SPIFFE_PI / m->nr)) / (1 + rz * rz);
  double *om = new double[limit];
  double omega = 1.0;
  for (long long n = 0; n < limit; n++) {
    om[n] = omega;
    if (n == 0)
      omega = 1.0 / (1 - rj * rj / 2);
    else
      omega = 1.0 / (1 - rj * rj * omega / 4);
  }
  cudaError_t e = dev_malloc(&w->omega, sizeof(double) * limit);
  if (e == cudaSuccess) e = cudaMemcpyAsync(w->omega, om, sizeof(double) * limit, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  delete[] om;
  w->omega_n = limit;
  return (int)e;
}

static int sum_region(const double *a, int rows, int cols, int P, int absval, Poisson64Work *w, double *out,
                      cudaStream_t s)
{
  dim3 block(BX, BY), grid((cols + BX - 1) / BX, (rows + BY - 1) / BY);
  if (grid.x * grid.y == 0) {
    cudaMemsetAsync(out, 0, sizeof(double), s);
    return 0;
  }
  k_region_sum<<<grid, block, 0, s>>>(a, rows, cols, P, absval, w->part);
  spiffe_note_launches(1);
  k_finish_sum<<<1, 1024, 0, s>>>(w->part, grid.x * grid.y, 1, out);
  spiffe_note_launches(1);
  return 0;
}

static int launch_sor(const DevMesh *m, Poisson64Work *w, double *Psi, const double *rhs, const int16_t *flags,
                      double accuracy, long long limit, PcState *st, long long *iters, DevCounts *cnt, cudaStream_t s)
{
  if (!w->part_n)
    return (int)cudaErrorInvalidValue;
  int rc = ensure_omega(m, w, limit, s);
  if (rc)
    return rc;
  // sum |rhs| over iz < nz, ir < nr-1 (poisson.c:333-336)
  if (rhs)
    sum_region(rhs, m->nz, m->nr - 1, m->pitch, 1, w, w->scalars + 4, s);
  else
    cudaMemsetAsync(w->scalars + 4, 0, sizeof(double), s);
  SorArgs a;
  a.Psi = Psi;
  a.rhs = rhs;
  a.flags = flags;
  a.omega = w->omega;
  a.a = 1 / (m->dz * m->dz);
  a.e = -2 * (1 / (m->dz * m->dz) + 1 / (m->dr * m->dr));
  a.crow = w->crow;
  a.drow = w->drow;
  const double c_axis = 1 / (m->dr * m->dr);
  a.c4_axis = 4 * c_axis;
  a.e2c_axis = a.e - 2 * c_axis;
  a.accuracy = accuracy;
  a.driving = w->scalars + 4;
  a.limit = limit;
  a.partials = w->part;
  a.bar_count = w->bar;
  a.bar_gen = w->bar + 1;
  a.st = st;
  a.iterations_out = iters;
  DevMesh mm = *m;
  cudaError_t e;
  // (end conditions set after the set-up move the update rows: the bands
  // follow those they were laid out for; and they divide by the diagonals
  // through their reciprocals, which gives the quotients' bits in div_by's
  // range)
  const int lo = m->left_bc == SPIFFE_DIRICHLET ? 0 : 1, hi = m->right_bc == SPIFFE_DIRICHLET ? m->nz - 1 : m->nz - 2;
  if (w->band_kernel && lo == w->band_lo && hi == w->band_hi && div_by_takes(-a.e) && div_by_takes(-a.e2c_axis)) {
    SorBand sb{w->band_R, w->band_H, 1 / a.e, 1 / a.e2c_axis, w->band_mem, w->band_xb, w->band_bar};
    e = cudaMemsetAsync(w->band_bar, 0, 32 * sizeof(unsigned long long), s);
    if (e != cudaSuccess)
      return (int)e;
    void *args[] = {&mm, &a, &sb, &cnt};
    if (w->band_cluster) {
      cudaLaunchAttribute at{};
      const cudaLaunchConfig_t c = sb_cluster_config(w->band_grid, w->band_smem, s, &at);
      e = cudaLaunchKernelExC(&c, w->band_kernel, args);
    } else {
      e = cudaLaunchCooperativeKernel(w->band_kernel, dim3(w->band_grid), dim3(SB_NT), args, w->band_smem, s);
    }
  } else {
    void *args[] = {&mm, &a, &cnt};
    e = cudaLaunchCooperativeKernel((void *)k_sor, dim3(w->sor_grid), dim3(RT), args, 0, s);
  }
  spiffe_note_launches(1);
  return (int)e;
}

// solve_poisson_cyl on device arrays; *iterations receives the reference's
// return value (n, or -1 when the limit was reached) after the stream syncs.
extern "C" int spiffe_sor64(const DevMesh *m, Poisson64Work *w, double *Psi, const double *rhs, const int16_t *flags,
                            double accuracy, long long limit, DevCounts *cnt, long long *iterations, cudaStream_t s)
{
  int rc = launch_sor(m, w, Psi, rhs, flags, accuracy, limit, nullptr, w->iters, cnt, s);
  if (rc)
    return rc;
  if (iterations) {
    cudaMemcpyAsync(iterations, w->iters, sizeof(long long), cudaMemcpyDeviceToHost, s);
    cudaStreamSynchronize(s);
  }
  return (int)cudaGetLastError();
}


// One add_poisson_correction pass (the interval test is the caller's).
extern "C" int spiffe_poisson_correction64(const DevMesh *m, const DevFields<double> *f, const DevBeam64 *b,
                                           DevCounts *cnt, long long np_bound, const PoissonHostOptions *o,
                                           Poisson64Work *w, Particles64Work *pw, bool ordered, cudaStream_t s)
{
  if (!w->part_n || (ordered && (!pw || !pw->keys || pw->capacity < np_bound)))
    return (int)cudaErrorInvalidValue;
  // the particles' own charge leaves Q (:190-242)
  const int stride = spiffe_smear_nodes(m), nodes = (m->nz + 1) * m->pitch;
  auto remove_charge = [&]() -> int {
    k_remove_charge<<<blocks_for(np_bound, RT), RT, 0, s>>>(*m, *f, *b, cnt, w->part, ordered ? pw->keys : nullptr,
                                                            ordered ? pw->vals : nullptr, (long)np_bound, stride, nodes);
    spiffe_note_launches(1);
    return ordered ? spiffe_ordered_add64(pw, stride * np_bound, nodes, f->Q, s) : 0;
  };
  dim3 block(BX, BY), grid((m->nr + 1 + BX - 1) / BX, (m->nz + 1 + BY - 1) / BY);
  const int nblk = grid.x * grid.y;
  // apparent charge, then the particles' own charge
  k_apparent_charge<<<grid, block, 0, s>>>(*m, *f, w->Az, w->Ari, w->Aro, 0, w->part);
  spiffe_note_launches(1);
  k_finish_sum<<<1, 1024, 0, s>>>(w->part, nblk, 2, w->scalars + 0);
  spiffe_note_launches(1);
  k_finish_sum<<<1, 1024, 0, s>>>(w->part + 1, nblk, 2, w->scalars + 1);
  spiffe_note_launches(1);
  if (o->space_charge && np_bound > 0) {
    const unsigned pb = blocks_for(np_bound, RT);
    if (int rc = remove_charge())
      return rc;
    k_finish_sum<<<1, 1024, 0, s>>>(w->part, (int)pb, 1, w->scalars + 2);
    spiffe_note_launches(1);
  } else {
    cudaMemsetAsync(w->scalars + 2, 0, sizeof(double), s);
  }
  sum_region(f->Q, m->nz, m->nr, m->pitch, 0, w, w->scalars + 3, s);
  const bool bound = o->error_charge_threshold > 0;
  if (bound)
    sum_region(f->Q, m->nz, m->nr, m->pitch, 1, w, w->scalars + 5, s);
  k_set_state<<<1, 1, 0, s>>>(w->st, w->scalars, w->scalars + 2, w->scalars + 3, o->space_charge);
  spiffe_note_launches(1);
  k_pc_decide<<<1, 1, 0, s>>>(w->st, o->error_charge_threshold, f->Q, m->nz, m->nr, m->pitch,
                              bound ? w->scalars + 5 : nullptr);
  spiffe_note_launches(1);
  k_scale_rhs<<<grid, block, 0, s>>>(*m, *f, w->volume, w->st);
  spiffe_note_launches(1);
  if (o->guess_code)
    { k_guess<<<grid, block, 0, s>>>(*m, *f, o->guess_code, w->st); spiffe_note_launches(1); }
  int rc = launch_sor(m, w, f->Psi, f->Q, f->flags, o->accuracy, o->maximum_iterations, w->st, w->iters, cnt, s);
  if (rc)
    return rc;
  k_subtract_gradient<<<grid, block, 0, s>>>(*m, *f, w->st);
  spiffe_note_launches(1);
  // the reference recomputes the apparent charge afterwards (:333-439)
  k_apparent_charge<<<grid, block, 0, s>>>(*m, *f, w->Az, w->Ari, w->Aro, 1, w->part);
  spiffe_note_launches(1);
  if (o->space_charge && np_bound > 0)
    if (int rc = remove_charge())
      return rc;
  return (int)cudaGetLastError();
}

// Downloads the last correction's report (synchronises the stream).
extern "C" int spiffe_poisson64_report(Poisson64Work *w, spiffe_poisson_report *rep, cudaStream_t s)
{
  PcState st;
  cudaMemcpyAsync(&st, w->st, sizeof(st), cudaMemcpyDeviceToHost, s);
  cudaError_t e = cudaStreamSynchronize(s);
  rep->ran = st.do_solve;
  rep->iterations = st.iterations;
  rep->Qreal = st.Qreal;
  rep->Qerror = st.Qerror;
  rep->Qsurface = st.Qsurface;
  rep->residual = st.residual;
  double drv = 0;
  cudaMemcpy(&drv, w->scalars + 4, sizeof(double), cudaMemcpyDeviceToHost);
  rep->driving = drv;
  return (int)e;
}

extern "C" int spiffe_imposed_field64(const DevMesh *m, const DevFields<double> *f, double factor, cudaStream_t s)
{
  dim3 block(BX, BY), grid((m->nr + 1 + BX - 1) / BX, (m->nz + 1 + BY - 1) / BY);
  k_imposed_field<<<grid, block, 0, s>>>(*m, *f, factor);
  spiffe_note_launches(1);
  return (int)cudaGetLastError();
}

// ----------------------------------------------- allocation-free SOR solve
//
// spiffe_gpu_solve_poisson_cyl_noalloc runs the same red-black SOR as
// spiffe_gpu_solve_poisson_cyl on device arrays the caller owns, for callers
// that must not allocate device memory: a host application whose device
// memory is owned by another framework's pool, which has reserved it and
// whose budget a cudaMalloc would break; or a control or real-time loop that
// forbids allocation after start-up so a solve can never fail for lack of
// memory or stall in the allocator.  Every piece of scratch the solve needs
// (the Chebyshev factors, the row coefficients, the block partial sums, the
// grid-barrier words and a counter block) lives in the fixed array below,
// which every GPU that loads this library holds until the process exits.

#define SPIFFE_NOALLOC_MAX_HALFSWEEPS 16384 // iteration_limit
#define SPIFFE_NOALLOC_MAX_NR 4096          // nr
#define SPIFFE_NOALLOC_MAX_PARTS 16384      // blocks of the |rhs| sum: ceil((nr-1)/32) * ceil(nz/8)
#define SPIFFE_NOALLOC_MAX_GRID 1024        // SOR blocks

struct NoallocScratch {
  double omega[SPIFFE_NOALLOC_MAX_HALFSWEEPS];
  double crow[SPIFFE_NOALLOC_MAX_NR + 1], drow[SPIFFE_NOALLOC_MAX_NR + 1];
  double part[SPIFFE_NOALLOC_MAX_PARTS];
  double sor_part[2 * SPIFFE_NOALLOC_MAX_GRID];
  double driving;
  long long iterations;
  unsigned bar[2];
  DevCounts cnt;
};

#define SPIFFE_NOALLOC_SCRATCH_BYTES (352u * 1024u)
static_assert(sizeof(NoallocScratch) <= SPIFFE_NOALLOC_SCRATCH_BYTES, "no-alloc scratch too small");

static __device__ __align__(256) unsigned char g_noalloc_scratch[SPIFFE_NOALLOC_SCRATCH_BYTES];

#include <cstdio>
#include <mutex>

namespace {
constexpr int NOALLOC_MAX_DEVICES = 64;
std::mutex g_noalloc_mutex;
int g_noalloc_grid[NOALLOC_MAX_DEVICES];
// host staging for the tables, static so the call allocates nothing
double g_noalloc_omega[SPIFFE_NOALLOC_MAX_HALFSWEEPS];
double g_noalloc_crow[SPIFFE_NOALLOC_MAX_NR + 1], g_noalloc_drow[SPIFFE_NOALLOC_MAX_NR + 1];
} // namespace

extern "C" int spiffe_set_error(int code, const char *msg);

extern "C" int spiffe_gpu_solve_poisson_cyl_noalloc(const spiffe_mesh *mesh, double *psi, const double *rhs,
                                                    const int16_t *flags, double accuracy, int64_t iteration_limit,
                                                    int64_t *iterations, void *stream)
{
  char msg[256];
  if (!mesh || !psi || !flags)
    return spiffe_set_error(-1, "null argument");
  if (accuracy <= 0)
    return spiffe_set_error(-1, "accuracy is <= 0 in solve_poisson_cyl");
  if (iteration_limit <= 1)
    return spiffe_set_error(-1, "iteration_limit is <= 1 in solve_poisson_cyl");
  const int nz = mesh->nz, nr = mesh->nr;
  if (nz < 3 || nr < 4)
    return spiffe_set_error(-1, "mesh too small (need nz>=3, nr>=4)");
  if (iteration_limit > SPIFFE_NOALLOC_MAX_HALFSWEEPS) {
    snprintf(msg, sizeof(msg), "iteration_limit %lld exceeds the allocation-free maximum of %d",
             (long long)iteration_limit, SPIFFE_NOALLOC_MAX_HALFSWEEPS);
    return spiffe_set_error(-1, msg);
  }
  if (nr > SPIFFE_NOALLOC_MAX_NR) {
    snprintf(msg, sizeof(msg), "nr=%d exceeds the allocation-free maximum of %d", nr, SPIFFE_NOALLOC_MAX_NR);
    return spiffe_set_error(-1, msg);
  }
  const dim3 sblock(BX, BY), sgrid((nr - 1 + BX - 1) / BX, (nz + BY - 1) / BY);
  if ((size_t)sgrid.x * sgrid.y > SPIFFE_NOALLOC_MAX_PARTS) {
    snprintf(msg, sizeof(msg), "mesh of %d x %d nodes exceeds the allocation-free maximum of %d sum blocks", nz, nr,
             SPIFFE_NOALLOC_MAX_PARTS);
    return spiffe_set_error(-1, msg);
  }
  cudaStream_t s = (cudaStream_t)stream;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NOALLOC_MAX_DEVICES)
    return spiffe_set_error(-2, "no current CUDA device");
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  // every call, with the caller's device and context current: the device
  // address of the scratch array (its host-side name is not a device
  // address).  The lookup allocates nothing, and repeating it keeps the
  // address right after a device reset or under another context.
  NoallocScratch *sc = nullptr;
  {
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) {
      snprintf(msg, sizeof(msg), "cudaGetSymbolAddress of the solver scratch failed: %s", cudaGetErrorString(e));
      return spiffe_set_error(-2, msg);
    }
    sc = (NoallocScratch *)p;
  }
  // the cooperative grid depends on the device only
  if (!g_noalloc_grid[dev]) {
    int sms = 0, per = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_sor, RT, 0);
    if (per > 4)
      per = 4;
    int grid = sms * (per > 0 ? per : 1);
    if (grid > SPIFFE_NOALLOC_MAX_GRID)
      grid = SPIFFE_NOALLOC_MAX_GRID;
    g_noalloc_grid[dev] = grid;
  }
  // the tables, with the expressions of the instance path (poisson.c:342-361)
  const double dz = mesh->dz, dr = mesh->dr;
  const double rz = dz / dr;
  const double rj = (cos(SPIFFE_PI / nz) + rz * rz * cos(SPIFFE_PI / nr)) / (1 + rz * rz);
  double omega = 1.0;
  for (long long n = 0; n < iteration_limit; n++) {
    g_noalloc_omega[n] = omega;
    omega = n == 0 ? 1.0 / (1 - rj * rj / 2) : 1.0 / (1 - rj * rj * omega / 4);
  }
  for (int ir = 0; ir <= nr; ir++) {
    if (ir != 0) {
      g_noalloc_crow[ir] = 1 / (dr * dr) * (1 + 1. / (2 * ir));
      g_noalloc_drow[ir] = 1 / (dr * dr) * (1 - 1. / (2 * ir));
    } else
      g_noalloc_crow[ir] = g_noalloc_drow[ir] = 1 / (dr * dr);
  }
  cudaError_t e = cudaMemcpyAsync(sc->omega, g_noalloc_omega, sizeof(double) * iteration_limit,
                                  cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(sc->crow, g_noalloc_crow, sizeof(double) * (nr + 1), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(sc->drow, g_noalloc_drow, sizeof(double) * (nr + 1), cudaMemcpyHostToDevice, s);
  // the array keeps the previous call's contents: clear what must start at zero
  if (e == cudaSuccess)
    e = cudaMemsetAsync(sc->bar, 0, sizeof(sc->bar), s);
  if (e == cudaSuccess)
    e = cudaMemsetAsync(&sc->cnt, 0, sizeof(DevCounts), s);
  if (e == cudaSuccess)
    e = cudaMemsetAsync(&sc->iterations, 0, sizeof(long long), s);
  if (e != cudaSuccess) {
    snprintf(msg, sizeof(msg), "staging the solver tables failed: %s", cudaGetErrorString(e));
    return spiffe_set_error(-2, msg);
  }
  DevMesh m{};
  m.nz = nz;
  m.nr = nr;
  m.pitch = nr + 1;
  m.zmin = mesh->zmin;
  m.zmax = mesh->zmax;
  m.rmax = mesh->rmax;
  m.dz = dz;
  m.dr = dr;
  m.dt = mesh->dt;
  m.lower_bc = mesh->lower_bc;
  m.upper_bc = mesh->upper_bc;
  m.right_bc = mesh->right_bc;
  m.left_bc = mesh->left_bc;
  m.modes = mesh->modes;
  // sum |rhs| over iz < nz, ir < nr-1 (poisson.c:333-336), as the instance path forms it
  if (rhs) {
    k_region_sum<<<sgrid, sblock, 0, s>>>(rhs, nz, nr - 1, nr + 1, 1, sc->part);
    spiffe_note_launches(1);
    k_finish_sum<<<1, 1024, 0, s>>>(sc->part, sgrid.x * sgrid.y, 1, &sc->driving);
    spiffe_note_launches(1);
  } else {
    cudaMemsetAsync(&sc->driving, 0, sizeof(double), s);
  }
  SorArgs a;
  a.Psi = psi;
  a.rhs = rhs;
  a.flags = flags;
  a.omega = sc->omega;
  a.a = 1 / (dz * dz);
  a.e = -2 * (1 / (dz * dz) + 1 / (dr * dr));
  a.crow = sc->crow;
  a.drow = sc->drow;
  const double c_axis = 1 / (dr * dr);
  a.c4_axis = 4 * c_axis;
  a.e2c_axis = a.e - 2 * c_axis;
  a.accuracy = accuracy;
  a.driving = &sc->driving;
  a.limit = iteration_limit;
  a.partials = sc->sor_part;
  a.bar_count = sc->bar;
  a.bar_gen = sc->bar + 1;
  a.st = nullptr;
  a.iterations_out = &sc->iterations;
  DevCounts *cnt = &sc->cnt;
  void *args[] = {&m, &a, &cnt};
  e = cudaLaunchCooperativeKernel((void *)k_sor, dim3(g_noalloc_grid[dev]), dim3(RT), args, 0, s);
  spiffe_note_launches(1);
  long long it = 0;
  unsigned err = 0;
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(&it, &sc->iterations, sizeof(it), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(&err, &sc->cnt.error, sizeof(err), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess)
    e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) {
    snprintf(msg, sizeof(msg), "allocation-free SOR failed: %s", cudaGetErrorString(e));
    return spiffe_set_error(-2, msg);
  }
  if (err & SPIFFE_DEV_ERR_BARRIER)
    return spiffe_set_error(-4, "allocation-free SOR: grid barrier timed out");
  if (iterations)
    *iterations = it;
  return 0;
}
