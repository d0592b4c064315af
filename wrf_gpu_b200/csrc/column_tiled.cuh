// Column kernel of one acoustic substep, level-parallel version.
//
// A block owns TX (16 or 32) adjacent columns of one row j and all levels.
// Its TY level lanes split the levels (lane l holds the NP positions l, l+TY,
// ...) for every part of advance_mu_t / advance_w / calc_p_rho that is
// independent across levels; only the four genuine column recurrences run
// serially, one thread per column, out of shared memory:
//   * dmdt = sum_k dnw*dvdxi            (dynamics/mu_t_advance.py:205)
//   * the ww prefix subtraction         (dynamics/mu_t_advance.py:229-237)
//   * the Thomas forward and back sweeps (core/advance_w.py:558-592)
// Every expression keeps the operation order of the thread-per-column form
// (and of the reference), so results are identical to it bit for bit.
//
// What bounds it: latency.  The access pattern alone reaches 6.2 TB/s (a
// probe with 20 loads in flight per thread); clock stamps showed a block
// spending its time on per-level chains -- a load behind the previous level's
// branch, a division's 113 cycles, a coefficient evicted from the 30 KB of L1
// that the shared arrays leave, the surface w on one lane, the row prefetches
// at ~60 cycles each.  So: positions unrolled (NP) with their loads issued
// together; inputs of a phase copied or loaded during the serial phase before
// it; the level coefficients in shared memory; straight-line division batches;
// the surface w formed by its own warp at the start; one prefetch per line;
// few positions (26 lanes) on 16 columns, two blocks per SM, so that one
// block's serial phases overlap the other's loads.
// 433 x 433 x 50: 0.776 -> 0.615 ms per launch (2.25 GB at 2.9 TB/s -> 2.04 GB at 3.3);
// 256 x 256 x 50: 0.286 -> 0.220 ms; 64 x 64 x 40: 29.5 -> 16.9 us.
#pragma once
#include "dycore_common.cuh"
#include "acoustic_kernels.cuh"
#include "column_shape.cuh"

namespace wg {

// Resident blocks per SM requested from the register allocator, by width.
#ifndef WG_COL_MINB16
#define WG_COL_MINB16 2
#endif
#ifndef WG_COL_MINB
#define WG_COL_MINB 1
#endif
// L2 prefetch of the block's input rows: 0 off, 1 on.
#ifndef WG_COL_PREFETCH
#define WG_COL_PREFETCH 1
#endif
constexpr int col_minb(int tx) { return tx == 16 ? WG_COL_MINB16 : WG_COL_MINB; }
// Levels per software-pipelined batch of the serial recurrences: the batch's
// shared-memory operands are loaded before its first store, so the loads
// overlap instead of each waiting behind the previous level's store.
#ifndef WG_COL_SU
#define WG_COL_SU 8
#endif
constexpr int COL_SU = WG_COL_SU;

// L2 prefetch of the rows (levels 0..nz) this block reads directly in its later
// phases, by the lanes that have nothing to do in the serial column sum (lane
// index `lane` of `nlanes`): one touched element per 128 bytes and the row's
// last.  (One bulk prefetch instruction per row took ~60 cycles each, which
// delayed the whole block.)
template <int TX>
__device__ __forceinline__ void column_prefetch(const Grid &g, const Acoustic &A, const ColArgs &c, int i0, int j,
                                                int lane, int nlanes) {
  const int nx = g.nx, nz = g.nz, plane = g.ny * nx;
  constexpr int LINES = TX / 16 + 1;
  for (int e = lane * TX + threadIdx.x; e < (nz + 1) * LINES; e += nlanes * TX) {
    const int k = e / LINES, part = e - k * LINES;
    const size_t f = (size_t)(unsigned)(k * plane + j * nx + min(i0 + min(part * 16, TX - 1), nx - 1));
    auto pf = [&](const double *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p + f)); };
    if (k < nz) {
      pf(A.theta_s);
      pf(A.c2a);
      pf(A.alt);
      pf(A.pm1);
    }
    pf(A.pt1);
    pf(A.ph);
    pf(A.ph_tend);
    pf(A.w);
    pf(A.rw_tend);
    pf(A.cqw);
    pf(A.a);
    pf(A.alpha);
    pf(A.gamma);
    if (c.damp_opt == 3) pf(A.w_save);
  }
}

// PIN: compile in the boundary cadence's ring-0 pins of mu / muts / muave and
// the work theta, and the ring-0 ph pin (cadence and nested child); off, the
// kernel carries no trace of them.
template <int TX, int NP, bool PIN = false>
__global__ void __launch_bounds__(TX * COL_TY, col_minb(TX)) k_column_tiled(Grid g, Acoustic A, ColArgs c,
                                                                             const double *dvdxi, const double *hdiv) {
  static_assert(TX == 16 || TX == 32, "a column block is 16 or 32 columns wide");
  // rows ty < R0 share warp 0 with the serial thread row ty == 0
  constexpr int R0 = 32 / TX;
  extern __shared__ double sm[];
  const int tx = threadIdx.x, ty = threadIdx.y, TY = blockDim.y;
  const int nx = g.nx, ny = g.ny, nz = g.nz, plane = ny * nx;
  const int ig = blockIdx.x * TX + tx;
  const int j = blockIdx.y;
  const bool valid = ig < nx;
  const int i = valid ? ig : nx - 1;  // spare columns shadow the last one and store nothing
  const int L = nz + 1;
  auto S = [&](int a, int k) -> double & { return sm[(a * L + k) * TX + tx]; };
  // array roles, in order of use:
  //   A0 dvdxi, then theta_1, then a      A4 t_tend, then old ph, then new ph
  //   A1 dnw dvdxi, ww increments, wd, w   A5 hdiv, then coef, then gamma
  //   A2 ww_1, then old w, then rhs       A6 t_2ave, then buoy
  //   A3 ww, then alpha                   A7 theta_w
  constexpr int A0 = 0, A1 = 1, A2 = 2, A3 = 3, A4 = 4, A5 = 5, A6 = 6, A7 = 7;
  const int c2d = j * nx + i;
  auto M = [&](int k) { return (size_t)(unsigned)(k * plane + c2d); };
  // position n of this lane: level / face ty + n*TY, clamped for the loads so
  // that they are issued together; only stores look at the true position
  auto pos = [&](int n) { return ty + n * TY; };
  auto kc = [&](int n) { return min(pos(n), nz - 1); };
  auto fc = [&](int n) { return min(pos(n), nz); };
  const double dts = c.dts;
  const double eps_p = 1.0 + c.epssm, eps_m = 1.0 - c.epssm;
  const bool active = !c.specified || (j >= 1 && j <= ny - 2 && i >= 1 && i <= nx - 2);

  __shared__ double s_dmdt[TX], s_mutend[TX], s_muts[TX], s_muave[TX];
  // (row nz of the level arrays A6 and A7 is free: the limiter's scale and the surface w)
  // The level coefficients: staged in shared memory (read from global memory
  // they are evicted from the small L1 that the shared arrays leave over, and
  // every phase then waits on L2 for them); columns too tall for that read
  // global memory.
  constexpr bool SM_MET = NP <= COL_MET_NP;
  enum { MET_DNW, MET_C1H, MET_C2H, MET_C1F, MET_C2F, MET_RDNW, MET_RDN, MET_FNM, MET_FNP };
  const double *const gmet[COL_NMET] = {g.dnw, g.c1h, g.c2h, g.c1f, g.c2f, g.rdnw, g.rdn, g.fnm, g.fnp};
  double *const smet = sm + COL_NARR * L * TX;
  if (SM_MET) {
    for (int k = ty * TX + tx; k <= nz; k += TY * TX) {
#pragma unroll
      for (int a = 0; a < COL_NMET; ++a)
        smet[a * L + k] = ld(gmet[a], (a == MET_C1F || a == MET_C2F) ? k : min(k, nz - 1));
    }
  }
  auto met = [&](int a, int k) { return SM_MET ? smet[a * L + k] : ld(gmet[a], k); };
  const double msfty = ld(g.msfty, c2d);
  const double mut = ld(A.mut, c2d);
  const double minv = ld(g.rmsfty, c2d);  // == 1.0 / msfty
  // 2-D inputs of the serial phases, loaded early so their latency overlaps P1
  double muts_in = 0.0, mu_in = 0.0, mu_tend_in = 0.0, muave_in = 0.0, ww_bot = 0.0, ww_top = 0.0;
  if (ty == 0) {
    muts_in = A.muts[c2d];
    muave_in = A.muave[c2d];
    mu_in = A.mu[c2d];
    mu_tend_in = (A.mu_tend != nullptr) ? ld(A.mu_tend, c2d) : 0.0;
    ww_bot = A.ww[M(0)];
    ww_top = A.ww[M(nz)];
  }
  // ---------------- P1: stage dvdxi -> A0; ww_1, theta_w, t_2ave, t_tend, hdiv in flight ----------------
#pragma unroll
  for (int n = 0; n < NP; ++n)
    if (pos(n) < nz) cp_async8(&S(A0, pos(n)), dvdxi + M(pos(n)));
  cp_async_commit();
#pragma unroll
  for (int n = 0; n < NP; ++n) {
    const int k = pos(n);
    if (k < nz) {
      cp_async8(&S(A2, k), A.ww_1 + M(k));
      cp_async8(&S(A7, k), A.theta_w + M(k));
      cp_async8(&S(A6, k), A.t2ave + M(k));
      cp_async8(&S(A4, k), A.t_tend + M(k));
      cp_async8(&S(A5, k), hdiv + M(k));
    }
  }
  cp_async_commit();
  if (ty == R0) {  // the surface w from the terrain slope
    auto HT = [&](int jj, int ii2) {
      jj = jj < 0 ? 0 : (jj > ny - 1 ? ny - 1 : jj);
      ii2 = ii2 < 0 ? 0 : (ii2 > nx - 1 ? nx - 1 : ii2);
      return div_rcp(ld(A.phb0, ix2(jj, ii2, nx)), G, RG);
    };
    const int nxu = nx + 1, nyv = ny + 1;
    const double msftx = ld(g.msftx, c2d);
    const double htc = HT(j, i);
    const double dy_n = HT(j + 1, i) - htc, dy_s = htc - HT(j - 1, i);
    const double dx_e = HT(j, i + 1) - htc, dx_w = htc - HT(j, i - 1);
    auto vcf = [&](int jv) {
      return g.cf1 * ld(A.v_1, ix3(0, jv, i, nyv, nx)) + g.cf2 * ld(A.v_1, ix3(1, jv, i, nyv, nx)) +
             g.cf3 * ld(A.v_1, ix3(2, jv, i, nyv, nx));
    };
    auto ucf = [&](int iu) {
      return g.cf1 * ld(A.u_1, ix3(0, j, iu, ny, nxu)) + g.cf2 * ld(A.u_1, ix3(1, j, iu, ny, nxu)) +
             g.cf3 * ld(A.u_1, ix3(2, j, iu, ny, nxu));
    };
    S(A7, nz) = msfty * 0.5 * g.rdy * (dy_n * vcf(j + 1) + dy_s * vcf(j)) +
               msftx * 0.5 * g.rdx * (dx_e * ucf(i + 1) + dx_w * ucf(i));
  }
  cp_async_wait<1>();
#pragma unroll
  for (int n = 0; n < NP; ++n)
    if (pos(n) < nz) S(A1, pos(n)) = ld(g.dnw, pos(n)) * S(A0, pos(n));
  __syncthreads();
  // ---------------- P2: column sum and 2-D mass updates (serial, ty == 0) ----------------
  if (ty == 0) {
    double dmdt = 0.0, mu_tend = mu_tend_in, scale = 1.0, muts = muts_in, muave = muave_in;
    if (active) {
      int k = 0;
      for (; k + COL_SU <= nz; k += COL_SU) {
        double t[COL_SU];
#pragma unroll
        for (int u = 0; u < COL_SU; ++u) t[u] = S(A1, k + u);
#pragma unroll
        for (int u = 0; u < COL_SU; ++u) dmdt = (k + u == 0) ? t[u] : dmdt + t[u];
      }
      for (; k < nz; ++k) {
        const double t = S(A1, k);
        dmdt = (k == 0) ? t : dmdt + t;
      }
      const double mu_work_old = muts_in - mut;
      const double mu_save = mu_in - mu_work_old;
      double mu_tendency = dmdt + mu_tend;
      if (c.specified) {
        const double floor_ = dmax(MIN_MUTS_PA, MIN_MUTS_FRACTION * mut);
        const double muts_old = mut + mu_work_old;
        const double raw = dts * mu_tendency;
        const double allowed = dmax(muts_old - floor_, 0.0);
        const double loss = -raw;
        const bool finite = isfinite(raw) && isfinite(muts_old);
        scale = (finite && (loss > allowed)) ? allowed / dmax(loss, 1.0) : (finite ? 1.0 : 0.0);
        scale = dmin(dmax(scale, 0.0), 1.0);
        mu_tendency = mu_tendency * scale;
        dmdt = dmdt * scale;
        mu_tend = mu_tend * scale;
      }
      const double mu_work_new = mu_work_old + dts * mu_tendency;
      muts = mut + mu_work_new;
      muave = 0.5 * ((1.0 + c.epssm) * mu_work_new + (1.0 - c.epssm) * mu_work_old);
      if (valid) {
        A.mu_o[c2d] = mu_save + mu_work_new;
        A.mudf_o[c2d] = mu_tendency;
        A.muts_o[c2d] = muts;
        A.muave_o[c2d] = muave;
      }
    } else if (PIN && c.cad) {
      // specified cadence: ring-0 mu', muts and muave pinned to the mu' leaf
      const double mu_pin = ring_target(c.cad_mu, 1, ny, nx, 0, j, i);
      muts = ld(c.mub, c2d) + mu_pin;
      muave = muts - mut;
      if (valid) {
        A.mu_o[c2d] = mu_pin;
        A.muts_o[c2d] = muts;
        A.muave_o[c2d] = muave;
      }
    }
    if (A.oop && valid && !active && !(PIN && c.cad)) {  // the frozen ring passes through
      A.mu_o[c2d] = mu_in;
      A.mudf_o[c2d] = A.mudf[c2d];
      A.muts_o[c2d] = muts;
      A.muave_o[c2d] = muave;
    }
    if (A.oop && valid) A.ww_o[M(nz)] = ww_top;
    s_dmdt[tx] = dmdt;
    s_mutend[tx] = mu_tend;
    S(A6, nz) = scale;
    s_muts[tx] = muts;
    s_muave[tx] = muave;
  }
  if (WG_COL_PREFETCH && ty >= R0) column_prefetch<TX>(g, A, c, blockIdx.x * TX, j, ty - R0, TY - R0);
  __syncthreads();
  // ---------------- P3: ww increments -> A1 (old ww of inactive columns -> A3) ----------------
  const double muts = s_muts[tx], muave = s_muave[tx];
  {
    const double dmdt = s_dmdt[tx], mu_tend = s_mutend[tx], scale = S(A6, nz);
#pragma unroll
    for (int n = 0; n < NP; ++n) {
      const int k = pos(n);
      if (k < nz) {
        double dv = S(A0, k);
        if (c.specified) dv = dv * scale;
        S(A1, k) = div_rcp(met(MET_DNW, k) * (met(MET_C1H, k) * dmdt + dv + met(MET_C1H, k) * mu_tend), msfty, minv);
      }
    }
    if (!active) {
      for (int k = ty; k <= nz; k += TY) S(A3, k) = A.ww[M(k)];
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  // ---------------- P4: ww prefix (serial) -> A3; theta_1 -> A0 in flight ----------------
#pragma unroll
  for (int n = 0; n < NP; ++n)
    if (pos(n) < nz) cp_async8(&S(A0, pos(n)), A.theta_s + M(pos(n)));
  cp_async_commit();
  if (ty == 0 && active) {
    double prev = ww_bot;
    S(A3, 0) = prev - S(A2, 0);
    int kk = 1;
    for (; kk + COL_SU <= nz; kk += COL_SU) {
      double r1[COL_SU], r2[COL_SU];
#pragma unroll
      for (int u = 0; u < COL_SU; ++u) {
        r1[u] = S(A1, kk - 1 + u);
        r2[u] = S(A2, kk + u);
      }
#pragma unroll
      for (int u = 0; u < COL_SU; ++u) {
        const double cur = prev - r1[u];
        S(A3, kk + u) = cur - r2[u];
        prev = cur;
      }
    }
    for (; kk < nz; ++kk) {
      const double cur = prev - S(A1, kk - 1);
      S(A3, kk) = cur - S(A2, kk);
      prev = cur;
    }
    S(A3, nz) = ww_top;
  }
  double c2a[NP], alt[NP], pt0[NP], pt1[NP];
#pragma unroll
  for (int n = 0; n < NP; ++n) {
    c2a[n] = ld(A.c2a, M(kc(n)));
    alt[n] = ld(A.alt, M(kc(n)));
    pt0[n] = ld(A.pt1, M(kc(n)));
    pt1[n] = ld(A.pt1, M(kc(n) + 1));
  }
  cp_async_wait<0>();
  __syncthreads();
  // ---------------- P5: theta update, t_2ave, wd -> A1, buoy -> A6, coef -> A5 ----------------
  const bool put = valid && (active || A.oop);
#pragma unroll
  for (int n = 0; n < NP; ++n) {
    const int k = pos(n);
    if (k <= nz) cp_async8(&S(A2, k), A.w + M(k));  // ww_1 was last read in P4
  }
#pragma unroll
  for (int n = 0; n < NP; ++n) {
    const int k = pos(n);
    if (k < nz) {
      const double ww_lo = S(A3, k), ww_hi = S(A3, k + 1);
      const double t1 = S(A0, k) - T0;
      const double c1h = met(MET_C1H, k), c2h = met(MET_C2H, k), rdnw = met(MET_RDNW, k);
      double thw = S(A7, k);
      const double wdtn_hi =
          (k + 1 < nz) ? ww_hi * (met(MET_FNM, k + 1) * (S(A0, k + 1) - T0) + met(MET_FNP, k + 1) * t1) : 0.0;
      const double wdtn_lo = (k >= 1) ? ww_lo * (met(MET_FNM, k) * t1 + met(MET_FNP, k) * (S(A0, k - 1) - T0)) : 0.0;
      const double tend = S(A5, k) + rdnw * (wdtn_hi - wdtn_lo);
      const double theta_i = thw + msfty * dts * S(A4, k);
      const double mass_h = c1h * muts + c2h, mass_t = c1h * mut + c2h;
      if (active) thw = theta_i - dts * msfty * tend;
      if (PIN && c.cad && !active)  // specified cadence: the ring-0 work theta whose finished theta is the leaf's
        thw = mass_h * (ring_target(c.cad_th, nz, ny, nx, k, j, i) - T0) - mass_t * t1;
      if (put || (PIN && c.cad && valid)) A.theta_o[M(k)] = thw;
      if (put) A.ww_o[M(k)] = ww_lo;
      S(A7, k) = thw;
      const double half = 0.5 * (eps_p * thw + eps_m * S(A6, k));
      const double dn[2] = {half + (c1h * muave) * T0, c2a[n] * rdnw};
      const double dd[2] = {mass_h * (T0 + t1), safe12(mass_t)};
      double dq[2];
      div_batch(dn, dd, dq);
      if (valid) A.t2ave_o[M(k)] = dq[0];
      S(A6, k) = c2a[n] * alt[n] * dq[0];
      S(A5, k) = dq[1];  // coef(k) for P7
      S(A1, k) = (0.5 * (ww_hi + ww_lo)) * rdnw * (pt1[n] - pt0[n]);
    }
    if (k <= nz) cp_async8(&S(A4, k), A.ph + M(k));  // t_tend was read above, by this thread
  }
  cp_async_commit();
  double pht[NP];
#pragma unroll
  for (int n = 0; n < NP; ++n) pht[n] = ld(A.ph_tend, M(fc(n)));
  cp_async_wait<0>();
  __syncthreads();
  // ---------------- P6: rhs -> A2 (faces 1..nz), old ph in A4 (faces 0..nz) ----------------
  double wo[NP], av[NP], al[NP], rt[NP], cq[NP];
  {
    const double c05gem = 0.5 * G * eps_m;
    double rn[NP], rd[NP], rq[NP];
#pragma unroll
    for (int n = 0; n < NP; ++n) {
      const int f = fc(n);
      wo[n] = S(A2, f);
      double r = dts * (pht[n] + c05gem * wo[n]);
      if (f > 0 && f < nz) r = r + (-(dts * (met(MET_FNM, f) * S(A1, f) + met(MET_FNP, f) * S(A1, f - 1))));
      rn[n] = msfty * r;
      rd[n] = met(MET_C1F, f) * mut + met(MET_C2F, f);
      rt[n] = ld(A.rw_tend, M(f));
      cq[n] = ld(A.cqw, M(f));
      av[n] = ld(A.a, M(f));
      al[n] = ld(A.alpha, M(f));
    }
    div_batch(rn, rd, rq);
#pragma unroll
    for (int n = 0; n < NP; ++n) {
      const int f = pos(n);
      if (f <= nz) S(A2, f) = (f == 0 || (f == nz && c.top_lid)) ? 0.0 : S(A4, f) + rq[n];
    }
  }
  __syncthreads();
  // ---------------- P7: explicit w -> A1; a -> A0, alpha -> A3 ----------------
  {
    const double c05dg = 0.5 * dts * G;
    const double dtsg = dts * G;
#pragma unroll
    for (int n = 0; n < NP; ++n) {
      const int f = pos(n);
      if (f <= nz) {
        double wn;
        if (f == 0) {
          wn = S(A7, nz);
        } else if (f < nz) {
          double rw = rt[n];
          if (c.w_damping == 1) {
            const double mf = met(MET_C1F, f) * mut + met(MET_C2F, f);
            const double vert_cfl = fabs(S(A3, f) / safe12(mf) * met(MET_RDNW, f) * dts);
            double damp = -sgn(wo[n]) * W_ALPHA * (vert_cfl - W_BETA) * mf;
            damp = (vert_cfl > W_BETA) ? damp : 0.0;
            rw = rw + damp;
          }
          wn = wo[n] + dts * rw;
          const double tA_u = S(A5, f) * (eps_p * (S(A2, f + 1) - S(A2, f)) + eps_m * (S(A4, f + 1) - S(A4, f)));
          const double tA_l = S(A5, f - 1) * (eps_p * (S(A2, f) - S(A2, f - 1)) + eps_m * (S(A4, f) - S(A4, f - 1)));
          const double tA = minv * cq[n] * (c05dg * met(MET_RDN, f)) * (tA_u - tA_l);
          const double tB = dtsg * minv * (met(MET_RDN, f) * (S(A6, f) - S(A6, f - 1)) - (met(MET_C1F, f) * muave));
          wn = wn + (tA + tB);
        } else {
          const int km1 = nz - 1;
          const double mhm = safe12(met(MET_C1H, km1) * mut + met(MET_C2H, km1));
          const double rdnw_t = met(MET_RDNW, km1);
          const double c2a_t = ld(A.c2a, M(km1)), alt_t = ld(A.alt, M(km1));
          const double t2a_t = A.t2ave_o[M(km1)];
          const double tA_top = -0.5 * dts * G / mhm * (rdnw_t * rdnw_t) * 2.0 * c2a_t *
                                (eps_p * (S(A2, nz) - S(A2, nz - 1)) + eps_m * (S(A4, nz) - S(A4, nz - 1)));
          const double tB_top = -dts * G * (2.0 * rdnw_t * c2a_t * alt_t * t2a_t + (met(MET_C1F, nz) * muave));
          const double w_top = wo[n] + dts * rt[n] + minv * (tA_top + tB_top);
          wn = c.top_lid ? 0.0 : w_top;
        }
        S(A1, f) = wn;      // wd(f) was last read in P6
        S(A0, f) = av[n];   // theta_1(f) was last read in P5
        S(A3, f) = al[n];   // ww(f) was last read above, by this thread
      }
    }
  }
  __syncthreads();
  // ---------------- P8: Thomas forward (serial); gamma -> A5 and the last phase's inputs in flight ----------------
#pragma unroll
  for (int n = 0; n < NP; ++n)
    if (pos(n) <= nz) cp_async8(&S(A5, pos(n)), A.gamma + M(pos(n)));
  cp_async_commit();
  double th[NP], pm1[NP];
#pragma unroll
  for (int n = 0; n < NP; ++n) {
    c2a[n] = ld(A.c2a, M(kc(n)));
    alt[n] = ld(A.alt, M(kc(n)));
    th[n] = ld(A.theta_s, M(kc(n)));
    pm1[n] = ld(A.pm1, M(kc(n)));
  }
  if (ty == 0) {
    double wf_prev = S(A1, 0);
    int f = 1;
    for (; f + COL_SU - 1 <= nz; f += COL_SU) {
      double r6[COL_SU], r0[COL_SU], r3[COL_SU];
#pragma unroll
      for (int u = 0; u < COL_SU; ++u) {
        r6[u] = S(A1, f + u);
        r0[u] = S(A0, f + u);
        r3[u] = S(A3, f + u);
      }
#pragma unroll
      for (int u = 0; u < COL_SU; ++u) {
        const double wf = (r6[u] - r0[u] * wf_prev) * r3[u];
        S(A1, f + u) = wf;
        wf_prev = wf;
      }
    }
    for (; f <= nz; ++f) {
      const double wf = (S(A1, f) - S(A0, f) * wf_prev) * S(A3, f);
      S(A1, f) = wf;
      wf_prev = wf;
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  // ---------------- P8b: Thomas back substitution (serial) ----------------
  if (ty == 0) {
    double ws_next = S(A1, nz);
    int f = nz - 1;
    for (; f - COL_SU + 1 >= 1; f -= COL_SU) {
      double r6[COL_SU], r5[COL_SU];
#pragma unroll
      for (int u = 0; u < COL_SU; ++u) {
        r6[u] = S(A1, f - u);
        r5[u] = S(A5, f - u);
      }
#pragma unroll
      for (int u = 0; u < COL_SU; ++u) {
        const double ws = r6[u] - r5[u] * ws_next;
        S(A1, f - u) = ws;
        ws_next = ws;
      }
    }
    for (; f >= 1; --f) {
      const double ws = S(A1, f) - S(A5, f) * ws_next;
      S(A1, f) = ws;
      ws_next = ws;
    }
  }
  __syncthreads();
  // ---------------- P9: Rayleigh damping, w out, phi finish -> A4 ----------------
  {
    double ws[NP], pn[NP], pd[NP], pq[NP];
#pragma unroll
    for (int n = 0; n < NP; ++n) ws[n] = S(A1, fc(n));
    if (c.damp_opt == 3 && c.dampcoef > 0.0) {
      const double dampmag = dts * c.dampcoef;
      const double hbot = div_rcp(ld(A.pt1, M(nz)), G, RG) - c.zdamp;
#pragma unroll
      for (int n = 0; n < NP; ++n) {
        const int f = pos(n);
        if (f >= 1 && f <= nz) {
          const double hk = div_rcp(ld(A.pt1, M(f)), G, RG);
          double dampwt = 0.0;
          if (hk >= hbot) {
            const double sv = sin(over_zdamp(0.5 * 3.141592653589793 * (hk - hbot), c));
            dampwt = dampmag * (sv * sv);
          }
          const double mf = met(MET_C1F, f) * mut + met(MET_C2F, f);
          ws[n] = (ws[n] - dampwt * mf * ld(A.w_save, M(f))) / (1.0 + dampwt);
        }
      }
    }
#pragma unroll
    for (int n = 0; n < NP; ++n) {
      pn[n] = msfty * 0.5 * dts * G * eps_p * ws[n];
      pd[n] = met(MET_C1F, fc(n)) * muts + met(MET_C2F, fc(n));
    }
    div_batch(pn, pd, pq);
#pragma unroll
    for (int n = 0; n < NP; ++n) {
      const int f = pos(n);
      if (f <= nz) {
        double phn = S(A2, f) + pq[n];
        if (f == 0) phn = S(A4, 0);
        if (PIN && !active && c.ph_pin)  // ring-0 work ph whose finished ph' is the leaf's (spec_bdyupdate_ph)
          phn = ring_target(c.cad_ph, nz + 1, ny, nx, f, j, i) - ld(c.ph_save, M(f));
        S(A4, f) = phn;
        if (valid) {
          A.ph_o[M(f)] = phn;
          A.w_o[M(f)] = ws[n];
        }
      }
    }
  }
  __syncthreads();
  // ---------------- P10: calc_p_rho with smdiv memory ----------------
  const double mu_work = muts - mut;
#pragma unroll
  for (int n = 0; n < NP; ++n) {
    const int k = pos(n);
    if (k < nz) {
      const double mass = met(MET_C1H, k) * muts + met(MET_C2H, k);
      const double safe = safe12(mass);
      const double mu_term = met(MET_C1H, k) * mu_work;
      const double t1 = th[n] - T0;
      const double ttr = T0 + t1;
      const double sttr = fabs(ttr) > 1.0e-6 ? ttr : 1.0e-6;
      const double dn[2] = {-(alt[n] * mu_term + met(MET_RDNW, k) * (S(A4, k + 1) - S(A4, k))),
                            alt[n] * (S(A7, k) - mu_term * t1)};
      const double dd[2] = {safe, safe * sttr};
      double dq[2];
      div_batch(dn, dd, dq);
      const double pp = c2a[n] * (dq[1] - dq[0]);
      if (valid) {
        A.p_o[M(k)] = pp + SMDIV * (pp - pm1[n]);
        A.pm1_o[M(k)] = pp;
        A.al_o[M(k)] = dq[0];
      }
    }
  }
}

}  // namespace wg
