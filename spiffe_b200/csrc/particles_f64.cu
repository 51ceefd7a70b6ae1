// spiffe_b200/csrc/particles_f64.cu -- plain FP64 particle kernels.
//
// Current deposition (space_charge.c:34-295), field gather (interpolateFields,
// advance_particles.c:622-890), the momentum kick and drift with loss tests
// (advance_particles.c:131-339), screen crossings (:362-434) and the removal
// of lost particles (:490-518), one thread per particle over the
// structure-of-arrays beam.  Arithmetic keeps the reference's expression
// order and the file is built with -fmad=false, so a particle's trajectory is
// bit-identical to the reference's given the same fields.  Deposition sums
// with FP64 atomics by default (order-dependent in the last bits) or, in the
// ordered mode, in particle order exactly as the serial reference does.
#include "modules.cuh"

#include "compact.cuh"

#include <algorithm>

namespace {

constexpr int T = 256;

__device__ __forceinline__ long trunc_l(double x) { return (long)x; }

// checkLossCode, advance_particles.c:31-65
__device__ int loss_code(const DevMesh &m, const int16_t *fl, long iz, long ir)
{
  const int P = m.pitch;
  const int16_t f0 = fl[node((int)iz, (int)ir, P)];
  if (f0 & SPIFFE_FL_IS_INSIDE)
    return 3;
  if (f0 & SPIFFE_FL_IS_SURFACE) {
    if (iz + 1 > m.nz)
      return 4;
    if (ir + 1 > m.nr)
      return 5;
    if (fl[node((int)iz + 1, (int)ir + 1, P)] & SPIFFE_FL_IS_METAL && fl[node((int)iz, (int)ir + 1, P)] & SPIFFE_FL_IS_METAL &&
        fl[node((int)iz + 1, (int)ir, P)] & SPIFFE_FL_IS_METAL)
      return 6;
  }
  return 0;
}

// interpolateFields, advance_particles.c:622-890.  E = Ez, Er, Ephi, Bz, Br, Bphi.
__device__ void gather(const DevMesh &m, const DevFields<double> &f, double z, double r, double *E)
{
  const long nz = m.nz, nr = m.nr;
  const int P = m.pitch;
  const double dz = m.dz, dr = m.dr, zmin = m.zmin;
  const bool longit = m.modes & SPIFFE_FL_LONGIT_INTERP, radial = m.modes & SPIFFE_FL_RADIAL_INTERP;
  const bool tm = m.modes & SPIFFE_FL_TM_FIELDS, te = m.modes & SPIFFE_FL_TE_FIELDS;
  const int16_t *fl = f.flags;
  long iz, ir, iz1, ir1;
  double fr, fl_, fa, fb;
  double Ez = 0, Er = 0, Ephi = 0, Bz = 0, Br = 0, Bphi = 0;
#define N(a, b) node((int)(a), (int)(b), P)
  // Ez and Br, :649-710
  if (longit) {
    fr = (z - zmin) / dz + 0.5;
    iz = trunc_l(fr);
    fr -= iz;
    fl_ = 1 - fr;
  } else {
    iz = trunc_l((z - zmin) / dz + 1);
    fl_ = 1;
    fr = 0;
  }
  if (radial) {
    fa = r / dr;
    ir = trunc_l(fa);
    fa -= ir;
    fb = 1 - fa;
  } else {
    ir = trunc_l(r / dr + 0.5);
    fa = 0;
    fb = 1;
  }
  if (iz >= 0 && iz < nz && ir >= 0 && ir < nr) {
    if ((iz1 = iz + 1) >= nz)
      iz1 = iz;
    if ((ir1 = ir + 1) >= nr)
      ir1 = ir;
    if (fl[N(iz, ir + 1)] & SPIFFE_FL_ER_ZERO && fl[N(iz, ir)] & SPIFFE_FL_ER_ZERO) {
      if (iz > 0 && (fl[N(iz - 1, ir)] || fl[N(iz - 1, ir + 1)]))
        iz = iz1;
      else
        iz1 = iz;
    } else if (fl[N(iz1, ir + 1)] & SPIFFE_FL_ER_ZERO && fl[N(iz1, ir)] & SPIFFE_FL_ER_ZERO) {
      iz1 = iz;
    }
    if (tm)
      Ez = fb * (fl_ * (f.Ez[N(iz, ir)] + f.EzImposed[N(iz, ir)]) + fr * (f.Ez[N(iz1, ir)] + f.EzImposed[N(iz1, ir)])) +
           fa * (fl_ * (f.Ez[N(iz, ir1)] + f.EzImposed[N(iz, ir1)]) + fr * (f.Ez[N(iz1, ir1)] + f.EzImposed[N(iz1, ir1)]));
    if (r != 0 && te)
      Br = fb * (fl_ * f.Br2[N(iz, ir)] + fr * f.Br2[N(iz1, ir)]) + fa * (fl_ * f.Br2[N(iz, ir1)] + fr * f.Br2[N(iz1, ir1)]);
  }
  // Er and Bz, :713-752
  if (longit) {
    fr = (z - zmin) / dz;
    iz = trunc_l(fr);
    fr -= iz;
    fl_ = 1 - fr;
  } else {
    iz = trunc_l((z - zmin) / dz + 0.5);
    fr = 0;
    fl_ = 1;
  }
  if (radial) {
    fa = r / dr + 0.5;
    ir = trunc_l(fa);
    fa -= ir;
    fb = 1 - fa;
  } else {
    ir = trunc_l(r / dr + 1);
    fa = 0;
    fb = 1;
  }
  if (iz >= 0 && iz < nz && ir >= 0) {
    if (ir >= nr)
      ir = nr - 1;
    iz1 = iz + 1;
    ir1 = ir + 1;
    if (fl[N(iz + 1, ir)] & SPIFFE_FL_EZ_ZERO && fl[N(iz, ir)] & SPIFFE_FL_EZ_ZERO)
      ir = ir1;
    else if (fl[N(iz + 1, ir + 1)] & SPIFFE_FL_EZ_ZERO && fl[N(iz, ir + 1)] & SPIFFE_FL_EZ_ZERO)
      ir1 = ir;
    if (r != 0 && tm)
      Er = fl_ * (fb * (f.Er[N(iz, ir)] + f.ErImposed[N(iz, ir)]) + fa * (f.Er[N(iz, ir1)] + f.ErImposed[N(iz, ir1)])) +
           fr * (fb * (f.Er[N(iz1, ir)] + f.ErImposed[N(iz1, ir)]) + fa * (f.Er[N(iz1, ir1)] + f.ErImposed[N(iz1, ir1)]));
    if (te)
      Bz = fl_ * (fb * f.Bz2[N(iz, ir)] + fa * f.Bz2[N(iz, ir1)]) + fr * (fb * f.Bz2[N(iz1, ir)] + fa * f.Bz2[N(iz1, ir1)]);
  }
  // Ephi, :754-786
  if (te && r != 0) {
    if (longit) {
      fr = (z - zmin) / dz;
      iz = trunc_l(fr);
      fr -= iz;
      fl_ = 1 - fr;
    } else {
      iz = trunc_l((z - zmin) / dz + 0.5);
      fr = 0;
      fl_ = 1;
    }
    if (radial) {
      fa = r / dr;
      ir = trunc_l(fa);
      fa -= ir;
      fb = 1 - fa;
    } else {
      ir = trunc_l(r / dr + 0.5);
      fa = 0;
      fb = 1;
    }
    if (iz >= 0 && iz < nz && ir >= 0 && ir < nr) {
      if ((iz1 = iz + 1) >= nz)
        iz1 = iz;
      if ((ir1 = ir + 1) >= nr)
        ir1 = ir;
      Ephi = fl_ * fb * f.Ephi[N(iz, ir)] + fr * fb * f.Ephi[N(iz1, ir)] + fl_ * fa * f.Ephi[N(iz, ir1)] +
             fr * fa * f.Ephi[N(iz1, ir1)];
    }
  }
  // Bphi at the E time level, :788-825
  if (tm) {
    if (longit) {
      fr = (z - zmin) / dz + 0.5;
      iz = trunc_l(fr);
      fr -= iz;
      fl_ = 1 - fr;
    } else {
      iz = trunc_l((z - zmin) / dz + 1);
      fr = 0;
      fl_ = 1;
    }
    if (radial) {
      fa = r / dr + 0.5;
      ir = trunc_l(fa);
      fa -= ir;
      fb = 1 - fa;
    } else {
      ir = trunc_l(r / dr + 1);
      fa = 0;
      fb = 1;
    }
    if (r != 0 && iz >= 0 && iz < nz) {
      if ((iz1 = iz + 1) >= nz)
        iz1 = iz;
      if (ir >= nr)
        ir = nr - 1;
      if ((ir1 = ir + 1) >= nr)
        ir1 = ir;
      Bphi = fl_ * fb * f.Bphi2[N(iz, ir)] + fr * fb * f.Bphi2[N(iz1, ir)] + fa * fl_ * f.Bphi2[N(iz, ir1)] +
             fr * fa * f.Bphi2[N(iz1, ir1)];
    }
  }
  // uniform fields, the on-axis expansion, switches, :828-857
  Ez += m.constE[0];
  Er += m.constE[1];
  Ephi += m.constE[2];
  Bz += m.constB[0];
  Br += m.constB[1];
  Bphi += m.constB[2];
  if (m.n_onaxis)
    onaxis_add(m, z, r, Ez, Er, Bphi);
  if (m.turn_off[0]) Ez = 0;
  if (m.turn_off[1]) Er = 0;
  if (m.turn_off[2]) Ephi = 0;
  if (m.turn_off[3]) Bz = 0;
  if (m.turn_off[4]) Br = 0;
  if (m.turn_off[5]) Bphi = 0;
  // solenoid fields on nodes, :859-875
  if (m.has_solenoid) {
    fr = (z - zmin) / dz;
    iz = trunc_l(fr);
    fa = r / dr;
    ir = trunc_l(fa);
    if (ir >= 0 && iz >= 0 && ir < nr && iz < nz) {
      fa -= ir;
      fb = 1 - fa;
      fr -= iz;
      fl_ = 1 - fr;
      Bz += fl_ * (fb * f.BzImposed[N(iz, ir)] + fa * f.BzImposed[N(iz, ir + 1)]) +
            fr * (fb * f.BzImposed[N(iz + 1, ir)] + fa * f.BzImposed[N(iz + 1, ir + 1)]);
      Br += fl_ * (fb * f.BrImposed[N(iz, ir)] + fa * f.BrImposed[N(iz, ir + 1)]) +
            fr * (fb * f.BrImposed[N(iz + 1, ir)] + fa * f.BrImposed[N(iz + 1, ir + 1)]);
    }
  }
#undef N
  E[0] = Ez;
  E[1] = Er;
  E[2] = Ephi;
  E[3] = Bz;
  E[4] = Br;
  E[5] = Bphi;
}


struct PushParams {
  double time, z_forces_start;
  double QoMC, stiffness;
  double tb_epm, tb_z_force, tb_r_force, tb_z_decel, tb_r_decel;
  int screen_momentum;
  LostLog lost;
};

__device__ void record(const DevScreen &s, long long step, long long *nb, long long *overflow, const DevBeam64 &b,
                       long ip, const double *q)
{
  const long long k = atomic_add_ll(nb, 1LL);
  if (k >= s.capacity) {
    atomic_add_ll(overflow, 1LL);
    return;
  }
  s.order[k] = (step << 32) | (long long)ip;
  for (int c = 0; c < SPIFFE_SCREEN_QUANS; c++)
    s.col[c][k] = q[c];
  s.rmin[k] = b.rmin[ip];
  s.rmax[k] = b.rmax[ip];
  s.zmin[k] = b.zmin[ip];
  s.zmax[k] = b.zmax[ip];
  s.generation[k] = b.generation[ip];
  s.particleID[k] = b.particleID[ip];
}

// Pre-kick momenta of the last particle, which the reference's screen loop
// reads through its function-scope pz0/pr0/r_pphi0 (advance_particles.c:79,
// :202-204, :383-385).
__global__ void k_snapshot_last(DevBeam64 b, DevCounts *cnt)
{
  const long long np = cnt->np;
  if (np > 0) {
    cnt->last_pz0 = b.pz[np - 1];
    cnt->last_pr0 = b.pr[np - 1];
    cnt->last_rpphi0 = b.r_pphi[np - 1];
  }
}

// advance_particles' per-particle loop (:131-339) and screen loop (:362-434).
__global__ void __launch_bounds__(T) k_push(DevMesh m, DevFields<double> f, DevBeam64 b, PushParams p,
                                             DevScreens scr, DevCounts *cnt, uint8_t *lost_flag, int32_t *lost_list)
{
  step_begin();
  const long ip = (long)blockIdx.x * T + threadIdx.x;
  const long np = (long)cnt->np;
  if (ip >= np)
    return;
  const double dt = m.dt, dz = m.dz, dr = m.dr, zmin = m.zmin, zmax = m.zmax, rmax = m.rmax;
  const long nz = m.nz, nr = m.nr;
  const int16_t *fl = f.flags;
  const bool forced = p.tb_epm && (p.tb_z_force || p.tb_r_force);
  double z, r, z0, r0s, vz, vr, pz, pr, r_pphi, vphi, gamma, pphi, adjust = 1, E[6];
  long iz, ir;
  bool lost = false, r_was_negative = false;
  uint64_t status = b.status[ip];
  double zmx = b.zmax[ip], zmn = b.zmin[ip], rmx = b.rmax[ip], rmn = b.rmin[ip];

  z = z0 = b.z[ip];
  r = r0s = b.r[ip];
  if (z > zmx) zmx = z;
  if (z < zmn) zmn = z;
  if (r > rmx) rmx = r;
  if (r < rmn) rmn = r;
  vz = b.vz[ip];
  vr = b.vr[ip];
  z += vz * dt;
  r += vr * dt;
  if (!(status & SPIFFE_PART_ACTIVE)) {
    // activation on entering the mesh, :167-189 (|r|/dr is bounded by nr
    // here; the reference would index past the flag array beyond it)
    iz = trunc_l((z - zmin) / dz);
    ir = trunc_l(fabs(r) / dr);
    if ((z >= zmin && z <= zmax && r <= rmax) && ir <= nr && !loss_code(m, fl, iz, ir)) {
      status |= SPIFFE_PART_ACTIVE;
      atomic_add_ll(&cnt->new_active, 1LL);
      b.t0[ip] = p.time;
      b.r0[ip] = r0s;
      b.z0[ip] = z0;
      if (iz > 0 && loss_code(m, fl, iz - 1, ir))
        adjust = (z - (iz * dz + zmin)) / (z - z0);
      else
        adjust = (z - zmin) / (z - z0);
      if (adjust > 1)
        adjust = 1;
    }
  }
  if (p.z_forces_start > zmin && p.z_forces_start < zmax) {
    if (z0 < p.z_forces_start) {
      if (z < p.z_forces_start)
        adjust = 0;
      else
        adjust = (z - p.z_forces_start) / (z - z0);
    }
  }
  const double pz0 = b.pz[ip], pr0 = b.pr[ip], rpp0 = b.r_pphi[ip];
  pz = pz0;
  pr = pr0;
  r_pphi = rpp0;
  vphi = b.vphi[ip];
  const bool active = status & SPIFFE_PART_ACTIVE;
  // loss tests, :211-236
  if (active && (z < zmin || z > zmax || r > rmax))
    lost = true;
  if (!lost && active) {
    iz = trunc_l((z - zmin) / dz);
    ir = trunc_l(fabs(r) / dr);
    if (iz > nz || ir > nr || iz < 0 || ir < 0)
      lost = true;
    else if (loss_code(m, fl, iz, ir))
      lost = true;
  }
  if (r < 0) {
    r *= -1;
    pr *= -1;
    r_was_negative = true;
  }
  if (!lost && active) {
    if (z > zmx) zmx = z;
    if (z < zmn) zmn = z;
    if (r > rmx) rmx = r;
    if (r < rmn) rmn = r;
  }
  if (!forced) {
    // momentum kick with the stored (old) velocities, :270-287
    if (active)
      gather(m, f, z, r, E);
    else
      E[0] = E[1] = E[2] = E[3] = E[4] = E[5] = 0;
    const double QoMC = p.QoMC, stiff = p.stiffness;
    pphi = (r ? r_pphi / r : 0);
    gamma = sqrt(pr * pr + pz * pz + pphi * pphi + 1);
    pr += adjust * dt * ((r ? pphi * pphi * SPIFFE_C_MKS / gamma / r : 0) + QoMC * (E[1] + vphi * E[3] - vz * E[5])) / stiff;
    pz += adjust * dt * QoMC * (E[0] + vr * E[5] - vphi * E[4]) / stiff;
    r_pphi += adjust * dt * QoMC * r * (E[2] + vz * E[4] - vr * E[3]) / stiff;
  } else {
    // forced test-beam acceleration, :289-311
    pphi = (r ? r_pphi / r : 0);
    gamma = sqrt(pr * pr + pz * pz + pphi * pphi + 1);
    pr += dt * ((r ? pphi * pphi * SPIFFE_C_MKS / gamma / r : 0));
    if (z <= p.tb_z_decel)
      pz += dt * p.tb_z_force;
    else {
      pz -= dt * p.tb_z_force;
      if (pz < 0)
        pz = 0;
    }
    if (r_was_negative)
      pr = 0;
    else if (r <= p.tb_r_decel)
      pr += dt * p.tb_r_force;
    else
      pr -= dt * p.tb_r_force;
  }
  // new velocities, setParticleVelocities :605-620
  double nvz, nvr, nvphi;
  if (r) {
    gamma = sqrt(pz * pz + pr * pr + (r_pphi / r) * (r_pphi / r) + 1);
    nvphi = SPIFFE_C_MKS * r_pphi / r / gamma;
  } else {
    gamma = sqrt(pz * pz + pr * pr + 1);
    nvphi = 0;
  }
  nvz = SPIFFE_C_MKS * pz / gamma;
  nvr = SPIFFE_C_MKS * pr / gamma;
  b.z[ip] = z;
  b.r[ip] = r;
  b.pz[ip] = pz;
  b.pr[ip] = pr;
  b.r_pphi[ip] = r_pphi;
  b.vz[ip] = nvz;
  b.vr[ip] = nvr;
  b.vphi[ip] = nvphi;
  b.zmax[ip] = zmx;
  b.zmin[ip] = zmn;
  b.rmax[ip] = rmx;
  b.rmin[ip] = rmn;
  if (lost) {
    status &= ~SPIFFE_PART_ACTIVE;
    status |= SPIFFE_PART_LOST;
    const long long slot = atomic_add_ll(&cnt->n_lost, 1LL);
    atomicMin(&cnt->first_lost, (long long)ip);
    lost_list[slot] = (int32_t)ip;
  }
  b.status[ip] = status;
  lost_flag[ip] = lost ? 1 : 0;
  if (lost && p.lost.rec) { // the loss epilogue, :437-487
    double pm = pz * pz + pr * pr;
    if (r)
      pm += (r_pphi / r) * (r_pphi / r);
    LostRecord rec{p.time, 0, 0, sqrt(pm), pz, pr, b.r0[ip], b.z0[ip], b.Q[ip], (long long)ip, p.lost.step,
                   b.particleID[ip], b.generation[ip], 0, 0, 0, 0.f, 0.f};
    rec.code = (int16_t)find_loss_coordinates(zmin, zmax, dz, dr, nr, fl, m.pitch, z0, r0s, z,
                                              r_was_negative ? -r : r, &rec.zLost, &rec.rLost);
    lost_append(p.lost, rec);
  }

  // screen crossings, :362-434
  if (scr.n) {
    const bool ref = p.screen_momentum == SPIFFE_SCREEN_REFERENCE;
    const double pz0s = ref ? cnt->last_pz0 : pz0, pr0s = ref ? cnt->last_pr0 : pr0;
    const double rpp0s = ref ? cnt->last_rpphi0 : rpp0;
    double r0 = r0s, q[SPIFFE_SCREEN_QUANS];
    for (int is = 0; is < scr.n; is++) {
      const DevScreen &s = scr.s[is];
      if (s.z_position <= z && s.z_position > z0 && s.direction == 1) {
        const double dtp = (s.z_position - z0) / vz;
        const double pphi_new = r ? r_pphi / r : 0;
        const double pphi0 = r0 ? rpp0s / r0 : 0;
        q[0] = r0 + vr * dtp;
        q[1] = pz0s + (pz - pz0s) / dt * dtp;
        q[2] = pr0s + (pr - pr0s) / dt * dtp;
        q[3] = pphi0 + (pphi_new - pphi0) / dt * dtp;
        q[4] = (p.time - dt + dtp);
        q[5] = b.Q[ip];
        q[6] = b.r0[ip];
        q[7] = b.t0[ip];
        record(s, scr.step, &cnt->screen_nb[is], &cnt->screen_overflow, b, ip, q);
      } else if (s.z_position >= z && s.z_position < z0 && s.direction == -1) {
        const double dtp = (s.z_position - z0) / vz;
        r0 += vr * dtp;
        q[0] = r0;
        q[1] = pz;
        q[2] = pr;
        q[3] = r0 ? r_pphi / r0 : 0;
        q[4] = (p.time - dt + dtp);
        q[5] = b.Q[ip];
        q[6] = b.r0[ip];
        q[7] = b.t0[ip];
        record(s, scr.step, &cnt->screen_nb[is], &cnt->screen_overflow, b, ip, q);
      }
    }
  }
}

// ------------------------------------------------------------ deposition
// add_particle_currents, space_charge.c:34-295, one thread per particle.
// Each particle's (up to) four node contributions per component are formed
// exactly as the reference forms them; they are either added with FP64
// atomics or written to a contribution list for the ordered reduction.

struct Contrib {
  int node[4];
  double val[4];
  int n;
};

__device__ void contrib_jz(const DevMesh &m, double z, double r, double v, double Q, double one_over, Contrib &c)
{
  const long nz = m.nz, nr = m.nr;
  const bool rsm = m.modes & SPIFFE_FL_RADIAL_SMEAR, lsm = m.modes & SPIFFE_FL_LONGIT_SMEAR;
  const double dz = m.dz, dr = m.dr, zmin = m.zmin;
  long iz, ir;
  double fp, fm, Jm, Jp;
  c.n = 0;
  ir = rsm ? trunc_l(r / dr) : trunc_l(r / dr + 0.5);
  iz = lsm ? trunc_l((z - zmin) / dz + 0.5) : trunc_l((z - zmin) / dz + 1.0);
  if (iz < 0 || iz > nz || ir < 0 || ir > nr)
    return;
  const double QVG = v * (Q * one_over);
  if (rsm) {
    fp = r / dr - ir;
    fm = 1 - fp;
  } else {
    fm = 1;
    fp = 0;
  }
  if (ir == 0) {
    Jm = 4 * fm * QVG;
    Jp = fp * QVG / (1.5 * 1.5 - 0.5 * 0.5);
  } else if (ir < nr - 1) {
    Jm = fm * QVG / ((ir + 0.5) * (ir + 0.5) - (ir - 0.5) * (ir - 0.5));
    Jp = fp * QVG / ((ir + 1.5) * (ir + 1.5) - (ir + 0.5) * (ir + 0.5));
  } else {
    Jm = 0;
    Jp = fp * QVG / ((ir + 0.5) * (ir + 0.5) - (ir - 0.5) * (ir - 0.5));
    ir--;
  }
  if (lsm) {
    if (iz == 0) {
      fp = 1;
      fm = 0;
    } else if (iz == nz) {
      fm = 1;
      fp = 0;
    } else {
      fp = (z - zmin) / dz + 0.5 - iz;
      fm = 1 - fp;
    }
  } else {
    fm = 1;
    fp = 0;
  }
  const int P = m.pitch;
  c.node[c.n] = (int)node((int)iz, (int)ir, P);
  c.val[c.n++] = fm * Jm;
  // row iz+1 exists only for iz < nz; at iz == nz its weight is zero (the
  // reference would index past the last row)
  if (lsm && iz < nz) {
    c.node[c.n] = (int)node((int)iz + 1, (int)ir, P);
    c.val[c.n++] = fp * Jm;
  }
  if (rsm) {
    c.node[c.n] = (int)node((int)iz, (int)ir + 1, P);
    c.val[c.n++] = fm * Jp;
    if (lsm && iz < nz) {
      c.node[c.n] = (int)node((int)iz + 1, (int)ir + 1, P);
      c.val[c.n++] = fp * Jp;
    }
  }
}

__device__ void contrib_jr(const DevMesh &m, double z, double r, double v, double Q, double one_over, Contrib &c)
{
  const long nz = m.nz, nr = m.nr;
  const bool rsm = m.modes & SPIFFE_FL_RADIAL_SMEAR, lsm = m.modes & SPIFFE_FL_LONGIT_SMEAR;
  const double dz = m.dz, dr = m.dr, zmin = m.zmin;
  long iz, ir;
  double fp, fm, Jm, Jp;
  c.n = 0;
  ir = rsm ? trunc_l(r / dr + 0.5) : trunc_l(r / dr + 1.0);
  iz = lsm ? trunc_l((z - zmin) / dz) : trunc_l((z - zmin) / dz + 0.5);
  if (iz < 0 || iz > nz || ir < 0 || ir >= nr)
    return;
  if (rsm) {
    fp = r / dr + 0.5 - ir;
    fm = 1 - fp;
  } else {
    fm = 1;
    fp = 0;
  }
  const double QVG = v * (Q * one_over);
  if (ir == 0) {
    Jm = 0;
    Jp = QVG;
  } else if (ir < nr - 1) {
    Jm = fm * QVG / ((double)ir * ir - (double)(ir - 1) * (ir - 1));
    Jp = fp * QVG / ((double)(ir + 1) * (ir + 1) - (double)ir * ir);
  } else {
    Jm = 0;
    ir--;
    Jp = QVG / ((double)(ir + 1) * (ir + 1) - (double)ir * ir);
  }
  if (lsm) {
    if (iz == nz) {
      fm = 1;
      fp = 0;
    } else {
      fp = (z - zmin) / dz - iz;
      fm = 1 - fp;
    }
  } else {
    fm = 1;
    fp = 0;
  }
  const int P = m.pitch;
  c.node[c.n] = (int)node((int)iz, (int)ir, P);
  c.val[c.n++] = fm * Jm;
  // row iz+1 exists only for iz < nz; at iz == nz its weight is zero (the
  // reference would index past the last row)
  if (lsm && iz < nz) {
    c.node[c.n] = (int)node((int)iz + 1, (int)ir, P);
    c.val[c.n++] = fp * Jm;
  }
  if (rsm) {
    c.node[c.n] = (int)node((int)iz, (int)ir + 1, P);
    c.val[c.n++] = fm * Jp;
    if (lsm && iz < nz) {
      c.node[c.n] = (int)node((int)iz + 1, (int)ir + 1, P);
      c.val[c.n++] = fp * Jp;
    }
  }
}

__device__ void contrib_jphi(const DevMesh &m, double z, double r, double v, double Q, double one_over, Contrib &c)
{
  const long nz = m.nz, nr = m.nr;
  const bool rsm = m.modes & SPIFFE_FL_RADIAL_SMEAR, lsm = m.modes & SPIFFE_FL_LONGIT_SMEAR;
  const double dz = m.dz, dr = m.dr, zmin = m.zmin;
  long iz, ir;
  double fp, fm, Jm, Jp;
  c.n = 0;
  ir = rsm ? trunc_l(r / dr) : trunc_l(r / dr + 0.5);
  iz = lsm ? trunc_l((z - zmin) / dz) : trunc_l((z - zmin) / dz + 0.5);
  if (iz < 0 || iz > nz || ir < 0 || ir > nr)
    return;
  if (rsm) {
    fp = r / dr - ir;
    fm = 1 - fp;
  } else {
    fm = 1;
    fp = 0;
  }
  const double QVG = v * (Q * one_over);
  if (ir == 0) {
    Jm = 4 * fm * QVG;
    Jp = fp * QVG / (1.5 * 1.5 - 0.5 * 0.5);
  } else if (ir < nr - 1) {
    Jm = fm * QVG / ((ir + 0.5) * (ir + 0.5) - (ir - 0.5) * (ir - 0.5));
    Jp = fp * QVG / ((ir + 1.5) * (ir + 1.5) - (ir + 0.5) * (ir + 0.5));
  } else {
    Jm = 0;
    Jp = fp * QVG / ((ir + 0.5) * (ir + 0.5) - (ir - 0.5) * (ir - 0.5));
    ir--;
  }
  if (lsm) {
    if (iz == nz - 1) {
      fp = 0;
      fm = 1 - fp;
    } else {
      fp = (z - zmin) / dz - iz;
      fm = 1 - fp;
    }
  } else {
    fm = 1;
    fp = 0;
  }
  const int P = m.pitch;
  c.node[c.n] = (int)node((int)iz, (int)ir, P);
  c.val[c.n++] = fm * Jm;
  // row iz+1 exists only for iz < nz; at iz == nz its weight is zero (the
  // reference would index past the last row)
  if (lsm && iz < nz) {
    c.node[c.n] = (int)node((int)iz + 1, (int)ir, P);
    c.val[c.n++] = fp * Jm;
  }
  if (rsm) {
    c.node[c.n] = (int)node((int)iz, (int)ir + 1, P);
    c.val[c.n++] = fm * Jp;
    if (lsm && iz < nz) {
      c.node[c.n] = (int)node((int)iz + 1, (int)ir + 1, P);
      c.val[c.n++] = fp * Jp;
    }
  }
}

// component: 0 Jz, 1 Jr, 2 Jphi.  keys/vals != nullptr selects the ordered
// mode: slot stride*ip+k receives contribution k (key = key0 + node, or `pad`) for
// every ip below the host's bound n_slots, so slots past the live np (after
// losses) hold padding rather than an earlier step's contributions.  stride
// is the most contributions the mesh's smearing gives (1, 2 or 4): the sort
// that follows costs by the slot.
__global__ void __launch_bounds__(T) k_deposit(DevMesh m, DevFields<double> f, DevBeam64 b, const DevCounts *cnt,
                                                int component, int *keys, double *vals, long long n_slots, int stride,
                                                int key0, int pad)
{
  step_begin();
  const long ip = (long)blockIdx.x * T + threadIdx.x;
  const long np = (long)cnt->np;
  Contrib c;
  c.n = 0;
  if (ip < np && b.status[ip] & SPIFFE_PART_ACTIVE) {
    const double one_over = 1 / (SPIFFE_PI * m.dz * (m.dr * m.dr));
    if (component == 0)
      contrib_jz(m, b.z[ip], b.r[ip], b.vz[ip], b.Q[ip], one_over, c);
    else if (component == 1)
      contrib_jr(m, b.z[ip], b.r[ip], b.vr[ip], b.Q[ip], one_over, c);
    else
      contrib_jphi(m, b.z[ip], b.r[ip], b.vphi[ip], b.Q[ip], one_over, c);
  }
  unsigned lo = 0xffffffffu, hi = 0u; // nodes this lane adds to, and their last column
  int col = 0;
  for (int k = 0; k < c.n; k++) {
    const unsigned nd = (unsigned)c.node[k];
    lo = min(lo, nd);
    hi = max(hi, nd);
    col = max(col, (int)(nd % (unsigned)m.pitch));
  }
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  col = __reduce_max_sync(0xffffffffu, col);
  if ((threadIdx.x & 31) == 0 && lo <= hi)
    widen_box(f.jbox, (int)(lo / (unsigned)m.pitch), (int)(hi / (unsigned)m.pitch), col);
  if (keys) {
    if (ip < n_slots)
      for (int k = 0; k < stride; k++) {
        keys[stride * ip + k] = k < c.n ? key0 + c.node[k] : pad;
        vals[stride * ip + k] = k < c.n ? c.val[k] : 0.0;
      }
    return;
  }
  double *J = component == 0 ? f.Jz : (component == 1 ? f.Jr : f.Jphi);
  for (int k = 0; k < c.n; k++)
    atomicAdd(J + c.node[k], c.val[k]);
}

// The same, unordered and without smearing, DT * DP particles a block, summed
// in shared memory before they go to J.  Atomics straight to J (k_deposit) come
// from every particle and, a bunch covering some hundred nodes, fall on a few
// slices of L2 (63 % of one slice's rate, 4 % of the average: 57 to 63 us a
// component and million particles).  A block whose nodes span more than DTILE
// adds directly; its nodes are then many.  A million particles of a
// bunch, Jz and Jr: 135 -> 42 us in random order, 210 -> 37 in the order of
// their cells, 37 -> 32 spread over the mesh.  Two blocks of 512 threads an SM:
// eight particles a thread left one (57 us).
constexpr int DT = 512, DP = 4, DTILE = DT * DP;

// tile[at] += v for the lanes with at >= 0.  An addition in shared memory is a
// loop of compare and swap that lanes of one address take in turn, so those of
// an address that SAME or more lanes share (particles in the order of their
// cells) are summed by shuffles first.
constexpr int SAME = 4;
__device__ __forceinline__ void tile_add(double *tile, int at, double v)
{
  const unsigned all = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned grp = __match_any_sync(all, at);
  bool single = at >= 0;
  for (unsigned many = __ballot_sync(all, at >= 0 && __popc(grp) >= SAME); many;) {
    const int first = __ffs(many) - 1;
    const unsigned g = __shfl_sync(all, grp, first);
    const bool in = g >> lane & 1;
    double x = in ? v : 0.0;
    for (int o = 16; o > 0; o >>= 1)
      x += __shfl_xor_sync(all, x, o);
    if (lane == first)
      atomicAdd(tile + at, x);
    if (in)
      single = false;
    many &= ~g;
  }
  if (single)
    atomicAdd(tile + at, v);
}

// The line is where a beam spread over the mesh, whose blocks find more nodes
// than a tile has, loses little: its blocks add straight to J all the same, later.
// Jz and Jr in us, straight to J / block sums (a bunch in random order, in cell
// order; spread, spread in the order of radii):
//                 3001 x 821                          301 x 83
//    32,768  10/17  11/19   9/12   9/15     52/21   66/16   8/16   8/18
//   131,072  23/17  27/19  10/12  10/23    192/21  246/16  13/17  13/16
//   196,608  32/17  40/18  12/12  12/23    286/21  366/16  17/17  17/17
//   262,144  41/17  53/18  13/13  13/23    378/21  486/16  21/17  21/16
// (601 x 165 between them.)  A bunch gains well below the line, on a coarse mesh
// from 16,384 particles; which of the two a beam is the host does not know.
constexpr long long DEPOSIT_TILE_MIN = 3 << 16;
__global__ void __launch_bounds__(DT, 2) k_deposit_tile(DevMesh m, DevFields<double> f, DevBeam64 b, const DevCounts *cnt,
                                                      int first, int last)
{
  step_begin();
  __shared__ double tile[DTILE];
  __shared__ int lim[4]; // first and last row, first and last column
  m.modes &= ~(unsigned)(SPIFFE_FL_RADIAL_SMEAR | SPIFFE_FL_LONGIT_SMEAR); // (none: folds their branches away)
  const long np = (long)cnt->np, base = (long)blockIdx.x * (DT * DP);
  if (base >= np)
    return;
  const int tid = threadIdx.x, P = m.pitch;
  const double one_over = 1 / (SPIFFE_PI * m.dz * (m.dr * m.dr));
  for (int comp = first; comp < last; comp++) {
    if (tid < 4)
      lim[tid] = tid & 1 ? -1 : 0x7fffffff;
    __syncthreads();
    int nd[DP], r0 = 0x7fffffff, r1 = -1, c0 = 0x7fffffff, c1 = -1;
    double v[DP];
    const double *vel = comp == 0 ? b.vz : comp == 1 ? b.vr : b.vphi;
#pragma unroll
    for (int k = 0; k < DP; k++) {
      const long ip = base + k * DT + tid;
      nd[k] = -1;
      v[k] = 0;
      if (ip < np && b.status[ip] & SPIFFE_PART_ACTIVE) {
        Contrib c;
        if (comp == 0)
          contrib_jz(m, b.z[ip], b.r[ip], vel[ip], b.Q[ip], one_over, c);
        else if (comp == 1)
          contrib_jr(m, b.z[ip], b.r[ip], vel[ip], b.Q[ip], one_over, c);
        else
          contrib_jphi(m, b.z[ip], b.r[ip], vel[ip], b.Q[ip], one_over, c);
        if (c.n) {
          nd[k] = c.node[0];
          v[k] = c.val[0];
          const int row = (int)((unsigned)nd[k] / (unsigned)P), col = nd[k] - row * P;
          r0 = min(r0, row);
          r1 = max(r1, row);
          c0 = min(c0, col);
          c1 = max(c1, col);
        }
      }
    }
    r0 = __reduce_min_sync(0xffffffffu, r0);
    r1 = __reduce_max_sync(0xffffffffu, r1);
    c0 = __reduce_min_sync(0xffffffffu, c0);
    c1 = __reduce_max_sync(0xffffffffu, c1);
    if ((tid & 31) == 0 && r0 <= r1) {
      atomicMin(lim, r0);
      atomicMax(lim + 1, r1);
      atomicMin(lim + 2, c0);
      atomicMax(lim + 3, c1);
    }
    __syncthreads();
    r0 = lim[0], r1 = lim[1], c0 = lim[2], c1 = lim[3];
    if (r0 <= r1) { // (the same for the whole block)
      double *J = comp == 0 ? f.Jz : comp == 1 ? f.Jr : f.Jphi;
      const int W = c1 - c0 + 1;
      const long long n = (long long)(r1 - r0 + 1) * W;
      if (tid == 0)
        widen_box(f.jbox, r0, r1, c1);
      if (n <= DTILE) {
        for (int t = tid; t < (int)n; t += DT)
          tile[t] = 0;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < DP; k++) {
          const int row = (int)((unsigned)max(nd[k], 0) / (unsigned)P);
          tile_add(tile, nd[k] >= 0 ? (row - r0) * W + nd[k] - row * P - c0 : -1, v[k]);
        }
        __syncthreads();
        for (int t = tid; t < (int)n; t += DT)
          if (tile[t] != 0) {
            const int row = t / W;
            atomicAdd(J + node(r0 + row, c0 + t - row * W, P), tile[t]);
          }
      } else {
#pragma unroll
        for (int k = 0; k < DP; k++)
          if (nd[k] >= 0)
            atomicAdd(J + nd[k], v[k]);
      }
    }
    __syncthreads(); // lim and the tile are used again
  }
}

// Ordered reduction: after a stable sort by node, each run of equal keys is
// summed in particle order starting from the array's current value, which is
// the reference's serial J[node] += ... sequence (space_charge.c:130-137).
// A run is a serial chain of FP64 additions by definition; what bounded the
// kernel was that one thread also loaded each value and key in turn (a run of
// a few thousand particles, the usual case of a bunch on a coarse mesh, at an
// L2 latency each).  A warp takes 32 entries: runs that end inside them are
// added by their first lanes together, and the one that goes on is added by
// the warp, which loads 32 entries ahead of the additions.  Those 32 are added
// without a condition: a predicated addition takes 19 cycles of the chain, a
// plain one 9 (the FP64 add's own latency is 8).  20,000 particles on a 301 x
// 83 gun mesh: 559 us -> 45 us a call; loads further ahead change nothing.
__global__ void __launch_bounds__(T) k_ordered_sum(const int *keys, const double *vals, long long n, int pad, double *J)
{
  const unsigned all = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const long long i = (long long)blockIdx.x * T + threadIdx.x;
  const int k = i < n ? keys[i] : pad;
  const double v = i < n ? vals[i] : 0.0;
  int before = __shfl_up_sync(all, k, 1);
  if (lane == 0)
    before = i > 0 && i < n ? keys[i - 1] : pad;
  const bool start = k != pad && (before != k || i == 0);
  const unsigned starts = __ballot_sync(all, start);
  if (!starts)
    return;
  double acc = start ? J[k] + v : 0.0;
  bool open = start;
  for (int d = 1; d < 32; d++) {
    const int kd = __shfl_down_sync(all, k, d);
    const double vd = __shfl_down_sync(all, v, d);
    open = open && lane + d < 32 && kd == k;
    if (open)
      acc += vd;
    if (!__any_sync(all, open))
      break;
  }
  // the last run of the 32 entries may go on behind them
  const int last = 31 - __clz(starts), kl = __shfl_sync(all, k, last);
  if (__shfl_sync(all, k, 31) == kl) {
    double a = __shfl_sync(all, acc, last);
    long long at = i + 32;
    int kk = at < n ? keys[at] : pad;
    double vv = at < n ? vals[at] : 0.0;
    unsigned in = __ballot_sync(all, kk == kl);
    while (in == all) {
      at += 32;
      const int kn = at < n ? keys[at] : pad; // (loads ahead of the additions)
      const double vn = at < n ? vals[at] : 0.0;
#pragma unroll
      for (int t = 0; t < 32; t++)
        a += __shfl_sync(all, vv, t);
      kk = kn;
      vv = vn;
      in = __ballot_sync(all, kk == kl);
    }
    const int m = __ffs(~in) - 1; // the run's last entries
    for (int t = 0; t < m; t++)
      a += __shfl_sync(all, vv, t);
    if (lane == last)
      acc = a;
  }
  if (start)
    J[k] = acc;
}

// ------------------------------------------------------------ compaction

// a group's loads before its stores: one after another they are 19 latencies
// (and all at once more registers than 1024 threads have)
__device__ __forceinline__ void move64(const DevBeam64 &b, int dst, int src)
{
  auto group = [&](auto... p) {
    auto store = [&](auto... v) { ((p[dst] = v), ...); };
    store(p[src]...);
  };
  group(b.Q, b.z, b.r, b.pz, b.pr, b.vz, b.vr);
  group(b.r_pphi, b.vphi, b.t0, b.r0, b.z0, b.rmin, b.zmin);
  group(b.rmax, b.zmax, b.generation, b.particleID, b.status);
}

// Reference compaction: the first lost index ends the beam.
__global__ void k_compact_reference(DevCounts *cnt, int oa)
{
  step_begin();
  const bool cut = cnt->n_lost && cnt->first_lost < cnt->np;
  end_push(cnt, cut ? cnt->np - cnt->first_lost : 0, cut ? cnt->first_lost : cnt->np, oa);
}

// Swap compaction: survivors at the end refill lost slots at the front, the
// j-th lost slot (ascending) taking the j-th survivor counted from the end.
// One launch, where flags, a scan, a map and the moves took six (3.9 us each of
// launching, the whole step of a small problem).  Few losses are the first
// block's, and the others end at once; of a burst every block takes a part (one
// block alone took 8 ns a loss and more: a push of two million that loses half
// 8.7 ms, now 1.0, as with the six launches; a million that lose 20,000 a push
// 0.59 -> 0.16).  In a burst the last block to have read the counts sets them for
// the next push.
constexpr int BURST = 1024; // losses
// blocks for a burst of at most n particles
unsigned burst_blocks(long long n)
{
  return n <= BURST ? 1u : (unsigned)std::min(64ll, std::max(2ll, (n + 16383) / 16384));
}
__global__ void __launch_bounds__(CT) k_compact_swap(DevBeam64 b, const uint8_t *lost, const int32_t *lost_list,
                                                      DevCounts *cnt, int32_t *holes, int32_t *donors, int oa)
{
  step_begin();
  // (without a burst the first block may have set the count to 0 already when
  // another reads it: no burst either way)
  const long long n_lost = *(volatile long long *)&cnt->n_lost, np = *(volatile long long *)&cnt->np;
  auto move = [&](int dst, int src) { move64(b, dst, src); };
  if (n_lost > BURST && gridDim.x > 1) {
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      if (atomicAdd(&cnt->compacting, 1u) == gridDim.x - 1) {
        cnt->compacting = 0;
        end_push(cnt, n_lost, np - n_lost, oa);
      }
    }
    compact_burst<true>((int)n_lost, (int)np, lost, holes, donors, move);
    return;
  }
  if (blockIdx.x > 0)
    return;
  if (n_lost > 0)
    compact_block<true>(n_lost, np, lost_list, holes, donors, [&](int i) { return lost[i] != 0; }, move);
  __syncthreads();
  if (threadIdx.x == 0)
    end_push(cnt, n_lost, np - n_lost, oa);
}

// The on-axis fields' extremes of the coming push (advance_particles.c:113-114)
__global__ void k_reset_onaxis(DevCounts *cnt)
{
  cnt->oa_min = INFINITY; // HUGE
  cnt->oa_max = -INFINITY;
}

} // namespace

// ------------------------------------------------------------ host entry

#include <cub/device/device_radix_sort.cuh>


extern "C" int spiffe_particles64_work(Particles64Work *w, long long capacity, bool ordered)
{
  cudaError_t e = cudaSuccess;
  if (w->capacity < capacity) {
    spiffe_particles64_work_free(w);
    cub::DeviceRadixSort::SortPairs(nullptr, w->cub_bytes, (int *)nullptr, (int *)nullptr, (double *)nullptr,
                                    (double *)nullptr, (int)(4 * capacity));
    const size_t n = (size_t)(capacity + 16);
    DeviceSlab m;
    m.add(&w->lost, n);
    m.add(&w->lost_list, n);
    m.add(&w->holes, n);
    m.add(&w->donors, n);
    m.add((char **)&w->cub_tmp, w->cub_bytes);
    e = m.make();
    if (e == cudaSuccess)
      w->capacity = capacity;
  }
  if (e == cudaSuccess && ordered && !w->keys) {
    const size_t n = 4 * (size_t)w->capacity;
    DeviceSlab m;
    m.add(&w->keys, n);
    m.add(&w->keys_alt, n);
    m.add(&w->vals, n);
    m.add(&w->vals_alt, n);
    e = m.make();
  }
  return (int)e;
}

extern "C" void spiffe_particles64_work_free(Particles64Work *w)
{
  dev_free(w->lost); // with the others of its slab
  dev_free(w->keys); // with the ordered sums' others
  *w = Particles64Work();
}

// add_particle_currents.  np_bound is a host-side upper bound on np.
extern "C" int spiffe_deposit64(const DevMesh *m, const DevFields<double> *f, const DevBeam64 *b, const DevCounts *cnt,
                                long long np_bound, bool ordered, Particles64Work *w, cudaStream_t s)
{
  if (np_bound <= 0)
    return 0;
  const unsigned nb = blocks_for(np_bound, T);
  const int nodes = (m->nz + 1) * m->pitch, stride = spiffe_smear_nodes(m);
  const int first = m->modes & SPIFFE_FL_TM_FIELDS ? 0 : 2, last = m->modes & SPIFFE_FL_TE_FIELDS ? 3 : 2;
  if (!ordered && stride == 1 && np_bound >= DEPOSIT_TILE_MIN) {
    if (last > first) {
      launch_next(k_deposit_tile, blocks_for(np_bound, DT * DP), DT, s, *m, *f, *b, cnt, first, last);
      spiffe_note_launches(1);
    }
    return (int)cudaGetLastError();
  }
  double *const J[3] = {f->Jz, f->Jr, f->Jphi};
  if (!ordered) {
    for (int comp = first; comp < last; comp++) {
      launch_next(k_deposit, nb, T, s, *m, *f, *b, cnt, comp, nullptr, nullptr, 0, stride, 0, nodes);
      spiffe_note_launches(1);
    }
    return (int)cudaGetLastError();
  }
  // The components' entries sorted and summed together where the buffers hold
  // them: J's components lie one behind the other, so a component is a range
  // of keys.  A call is latency (two passes of the sort, the longest run's
  // additions), which two components then share: 20,000 particles on 301 x
  // 83, 75 -> 38 us a component.
  const long long per = (long long)stride * np_bound, step = last - first > 1 ? J[first + 1] - J[first] : nodes;
  const int together = (last - first) * stride <= 4 && step >= nodes && (last - first) * step < 0x7fffffff ? last - first : 1;
  // (components after the first go to places reckoned from the buffers' start)
  if (!w->keys || together * per > 4 * w->capacity)
    return (int)cudaErrorInvalidValue;
  for (int comp = first; comp < last; comp += together) {
    const int pad = together > 1 ? (int)(together * step) : nodes;
    for (int k = 0; k < together; k++) {
      launch_next(k_deposit, nb, T, s, *m, *f, *b, cnt, comp + k, w->keys + k * per, w->vals + k * per, np_bound, stride,
                  (int)(k * step), pad);
      spiffe_note_launches(1);
    }
    if (int rc = spiffe_ordered_add64(w, together * per, pad, J[comp], s))
      return rc;
  }
  return (int)cudaGetLastError();
}

extern "C" int spiffe_ordered_add64(Particles64Work *w, long long n, int nodes, double *dst, cudaStream_t s)
{
  if (n <= 0)
    return 0;
  if (!w->keys || n > 4 * w->capacity)
    return (int)cudaErrorInvalidValue;
  // stable LSD radix sort keeps entry order inside each node's run, over the
  // bits that nodes and the pad key (one past the last node) have
  int bits = 1;
  while ((1ll << bits) <= nodes)
    bits++;
  size_t bytes = w->cub_bytes;
  cudaError_t e = cub::DeviceRadixSort::SortPairs(w->cub_tmp, bytes, w->keys, w->keys_alt, w->vals, w->vals_alt,
                                                  (int)n, 0, bits, s);
  if (e != cudaSuccess)
    return (int)e;
  k_ordered_sum<<<blocks_for(n, T), T, 0, s>>>(w->keys_alt, w->vals_alt, n, nodes, dst);
  spiffe_note_launches(1);
  return (int)cudaGetLastError();
}


namespace {
// interpolateFields at n points (zr[2i], zr[2i+1]): the first ncomp of
// Ez, Er, Ephi, Bz, Br, Bphi into E[ncomp*i ...]
__global__ void k_gather_points64(DevMesh m, DevFields<double> f, const double *zr, int n, int ncomp, double *E)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  double e[6];
  gather(m, f, zr[2 * i], zr[2 * i + 1], e);
  for (int c = 0; c < ncomp; c++)
    E[(size_t)ncomp * i + c] = e[c];
}
} // namespace

extern "C" int spiffe_gather_points64(const DevMesh *m, const DevFields<double> *f, const double *zr, int n, int ncomp,
                                      double *E, cudaStream_t s)
{
  if (n <= 0)
    return 0;
  k_gather_points64<<<blocks_for(n, 128), 128, 0, s>>>(*m, *f, zr, n, ncomp < 6 ? ncomp : 6, E);
  spiffe_note_launches(1);
  return (int)cudaGetLastError();
}

// advance_particles: snapshot, push with screens, then compaction.
extern "C" int spiffe_push64(const DevMesh *m, const DevFields<double> *f, const DevBeam64 *b, const PushHostParams *hp,
                             const DevScreens *scr, DevCounts *cnt, long long np_bound, Particles64Work *w, cudaStream_t s)
{
  if (np_bound > w->capacity)
    return (int)cudaErrorInvalidValue;
  if (m->n_onaxis) {
    k_reset_onaxis<<<1, 1, 0, s>>>(cnt);
    spiffe_note_launches(1);
  }
  const int oa = !m->n_onaxis;
  if (np_bound <= 0 && oa && w->met_none)
    return 0; // no particle, and nothing to reset: an empty push changes no count
  w->met_none = oa;
  if (np_bound > 0) {
    PushParams p{hp->time, hp->z_forces_start, hp->QoMC, hp->stiffness, hp->tb_epm, hp->tb_z_force,
                 hp->tb_r_force, hp->tb_z_decel, hp->tb_r_decel, hp->screen_momentum, hp->lost};
    if (scr->n && hp->screen_momentum == SPIFFE_SCREEN_REFERENCE)
      { k_snapshot_last<<<1, 1, 0, s>>>(*b, cnt); spiffe_note_launches(1); }
    launch_next(k_push, blocks_for(np_bound, T), T, s, *m, *f, *b, p, *scr, cnt, w->lost, w->lost_list);
    spiffe_note_launches(1);
  }
  if (hp->compaction == SPIFFE_COMPACT_REFERENCE || np_bound <= 0)
    launch_next(k_compact_reference, 1, 1, s, cnt, oa);
  else
    launch_next(k_compact_swap, burst_blocks(np_bound), CT, s, *b, w->lost, w->lost_list, cnt, w->holes, w->donors, oa);
  spiffe_note_launches(1);
  return (int)cudaGetLastError();
}
