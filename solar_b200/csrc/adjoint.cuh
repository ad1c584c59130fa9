// adjoint.cuh -- discrete adjoint of the time step (sm_100a).
//
// The forward step is linear in the state: per 2N-RK stage s (timestep.f90:64-69)
//     w_s = alpha_s w_{s-1} + dt L(q_{s-1}) ,   q_s = q_{s-1} + beta_s w_s
// with L = SPONGE o BC_RHS o COMPUTE_RHS, then q_{n+1} = F(q_5) (FILTER_EXP).  Its exact
// transpose, stage by stage in reverse, is
//     mu_s = lw_s + beta_s lq_s ;  lq_{s-1} = lq_s + dt L^T(mu_s) ;  lw_{s-1} = alpha_s mu_s
// and the gradient of a misfit with respect to a per-point sound-speed perturbation dc
// (c -> c + dc enters only r_p = -c^2 rho0 div v, compute_rhs_acoustic.f90:134) gathers
//     g += dt (-2 c rho0 div(v_{s-1})) mu_s^p            (0 on the BC planes).
// L^T is applied in two kernels:
//   adj_stage  mu, the BC mask, the pointwise terms, the sponge, g, and the transposed
//              derivatives of the coefficient-weighted fields: -D_xi and -D_eta with zero
//              halos (the DRP stencil is antisymmetric) and the radial transpose with its
//              one-sided (Tam-Dong) rows, on the interior and on the ghost frame -- the frame
//              values are the adjoints of the neighbour faces' ghost values;
//   adj_edge   the transpose of the edge exchange: each source-line point gathers the ghost
//              adjoints that used it, with the same folded coefficients.
// FILTER_EXP^T runs fused (adj_filter_kernel), its ghost-frame adjoints in a small kernel of
// their own, then the same scatter.
#pragma once

#include "kernels.cuh"

namespace solar {

// Fused transposed stage (pointwise part + transposed stencils in one pass).  The register
// lambda_w of the recursion above is never stored: with mu_s = lw_s + beta_s lq_s the
// recursion is
//     lq_{s-1} = lq_s + dt L^T(mu_s) ,   mu_{s-1} = alpha_s mu_s + beta_{s-1} lq_{s-1} ,
// so the buffers hold lambda_q and mu, and only mu (whose neighbours the stencils read) comes
// with a halo.  The step's first transposed stage (s = 5, where lw = 0) forms mu = beta lq from
// lambda_q alone; its last (s = 1) writes no mu.
//
// A CTA owns a TX x TY column tile of one face and marches the planes of its chunk (plus three
// planes on either side for the radial window).  Each thread owns V consecutive points of a row
// (V = 16 bytes / sizeof(T)).  Planes stream in through TMA tile loads into a ring of
// shared-memory slots, each guarded by an mbarrier: for a plane of the chunk the boxes of mu
// (tile plus a 4-column / 3-row halo) of v_xi, v_eta, p and rho, the tile of v_r, the lambda_q
// tiles, the c^2 box, the stored divergence, the gradient accumulator and the row of radial
// coefficients; for the three
// extra planes on either side the tiles of p, v_r, rho and c^2.  Per plane the kernel forms the
// coefficient-weighted volumes X1, X2 (on the tile and its xi halo) and Y1, Y2 (tile and eta
// halo) in shared memory (zero outside the face and on the BC planes; every thread takes its
// own vector and at most one halo vector), and after one barrier applies -D_xi / -D_eta.  The
// exchange arrays are double-buffered and a slot is read before the barrier only (behind a fence:
// most of what is read stays in registers), so that one barrier per plane serves both and thread 0
// refills the slot right after it.  The banded
// radial transpose adds each plane's facr * R1, facr * R2 to the partial outputs of the planes
// m-3 .. m+3, held in registers; a plane is complete three iterations later.  The one-sided
// rows of the radial stencil (planes 1, 2, nr-3, nr-2; planes 0 and nr-1 carry zero) reach the
// seven planes at each end: a chunk that holds some of them reads those rows' points itself.
// Edge tiles also write the ghost-frame adjoints.  Inputs (lambda_q, mu) and outputs are
// distinct buffers: neighbouring CTAs read the inputs' halos.
template <typename T>
struct AdjStageArgs {
  CUtensorMap mB3;        // boxes (TX+8) x (TY+6) of mu (of lambda_q in the first stage): (rho,) v_xi, v_eta
  CUtensorMap mB;         // box of p
  CUtensorMap mM;         // tiles TX x TY of the same buffer: v_r; v_r, p
  CUtensorMap mM2;
  CUtensorMap mQ;         // tiles TX x TY of all fields of lambda_q (not in the first stage)
  CUtensorMap mC2, mC2t;  // boxes and tiles of the compact c^2 (when present; zero outside the face)
  CUtensorMap mDiv;       // tiles TX x TY of the compact stored divergence (when present)
  CUtensorMap mGrad;      // tiles TX x TY of the gradient accumulator (double, when present)
  const T* mu;            // the buffer of mB
  T* lout;
  T* muout;               // nullptr in the last stage
  const T* div;           // compact stage-input divergence, or nullptr
  const T* c2;
  double* grad;           // sum over the stages of dt rho0 div mu_p (grad_scale_kernel: -2 c)
  const T* met;
  const T* radT;          // [nr][16]: the radial rows of a plane together (through the ring)
  WaitCtl wc;             // error word and bound of the ring waits
  Geom g;
  T alpha, beta, beta_next, dt, inv_dxi;   // mu = beta * box (1 but in the first stage)
  int first, keep, kchunk;
};

// What bounds it: the latency of a plane's loads.  Requests count as much as bytes: with one TMA
// request per field (14 per plane in double) a reverse step at 6 x 96^3 took 2045 us in double and
// 850 in float, with the fields of one shape in one 4-D request (8 per plane) 1681 and 838.  Two
// slots keep two CTAs per SM in double (110 KB each) and four in float (52 KB).  The form before
// (one point per thread, lambda_w and lambda_q boxes, two barriers per plane, a kernel of its own
// for the one-sided rows) took 2163 and 1198.
constexpr int kAdjRing = 2;

// Rounding.  dt L^T(mu) is small against lambda_q, so its terms are summed up before lambda_q comes
// in wherever registers allow, and what has to be added to the large sum later is added in as few
// parts as possible.  Error of lambda after 1 / 20 reverse steps in float against double, 6 x 48^2 x
// 33 and 6 x 96^3: 1.12e-7 / 2.84e-7 and 1.20e-7 / 3.23e-7; with lambda_q first and every plane's radial
// term added to it by itself 1.53e-7 / 3.42e-7 and 1.65e-7 / 4.15e-7.  In float lambda_q of p, v_xi and
// v_eta waits for the terms behind the barrier, and a plane's radial term of p for the next plane's
// (a step takes 0.3% less with four fields, 2.6% less with five, mean over ten grids from 6 x 64^3
// to 6 x 128^3).  In double the registers are used up: the same costs 5-30%, so there lambda_q
// comes in with the pointwise terms and the three later radial terms one by one.
template <typename T>
struct AdjSums {
  static constexpr bool late = sizeof(T) == 4;
};

template <typename T, int TX, int TY, bool HAS_RHO>
struct AdjLayout {
  static constexpr int V = Vec16<T>::V, NTH = TX / V * TY;
  static constexpr int PW = TX + 8, YH = TY + 6, PB = PW * YH, OB = TX * TY;
  static constexpr int NB = HAS_RHO ? 4 : 3, NF = NB + 1;
  static constexpr size_t P_BYTES = align128(PB * sizeof(T));
  static constexpr size_t O_BYTES = align128(OB * sizeof(T));
  // a chunk plane: boxes of mu [(rho,) v_xi, v_eta] as one load, [p], the tile of v_r, the
  // lambda_q tiles of every field in storage order as one load; an extra plane: tiles [v_r, p]
  // as one load, [rho], from the slot's start
  static constexpr size_t PBOX = align128((NB - 1) * PB * sizeof(T)), VR = PBOX + P_BYTES;
  static constexpr size_t LQ = VR + O_BYTES, C2 = LQ + NF * O_BYTES;
  static_assert(OB * sizeof(T) % 128 == 0, "tiles of one load follow each other");
  static constexpr size_t DIV = C2 + P_BYTES, GRAD = DIV + O_BYTES, RAD = GRAD + align128(OB * sizeof(double));
  static constexpr size_t SLOT = align128(RAD + 16 * sizeof(T));
  static constexpr int XB = TY * PW, YB = YH * TX;                  // exchange arrays
  static constexpr size_t EX = kAdjRing * SLOT;                     // [2][X1, X2, Y1, Y2]
  static constexpr size_t EX_BYTES = 2 * (XB + YB) * sizeof(T);
  static constexpr size_t ONE = EX + 2 * EX_BYTES;                  // one-sided rows, [4][NTH] vectors
  static constexpr size_t HELD = ONE + (size_t)4 * NTH * 16;        // a plane's radial term of p (AdjSums)
  static constexpr size_t BAR = HELD + (AdjSums<T>::late ? (size_t)NTH * 16 : 0);
  static constexpr size_t TOTAL = BAR + kAdjRing * sizeof(uint64_t);
};

template <typename T, int TX, int TY, bool HAS_RHO>
__global__ void __launch_bounds__(TX / Vec16<T>::V * TY) adj_stage_kernel(const __grid_constant__ AdjStageArgs<T> a) {
  using L = AdjLayout<T, TX, TY, HAS_RHO>;
  constexpr int V = L::V, NT = TX / V, PW = L::PW, YH = L::YH;
  constexpr int QV = 4 / V;                          // vectors in the 4-column margin of a box
  constexpr int NETA = 6 * NT, NXI = 2 * QV * TY;    // halo vectors
  constexpr int NV = (V + 8) / V;                    // vectors covering columns c-4 .. c+V+3
  constexpr bool LATE = AdjSums<T>::late;
  constexpr int PBs = L::PB, OBs = L::OB, R0 = HAS_RHO ? 1 : 0;   // storage slots: (rho,) v_xi, v_eta, v_r, p
  static_assert(NETA + NXI <= L::NTH, "one halo vector per thread");
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR);
  const Geom& g = a.g;
  const int n = g.n, nr = g.nr;
  const long long P2 = (long long)n * n;
  const int tiles_x = n / TX;
  const int i0 = (blockIdx.x % tiles_x) * TX, j0 = (blockIdx.x / tiles_x) * TY;
  const int face = blockIdx.z;
  const int kb = blockIdx.y * a.kchunk, ke = min(nr, kb + a.kchunk);
  if (kb >= nr) return;
  const int cx = threadIdx.x, ty = threadIdx.y, tid = ty * NT + cx;
  const int sRho = g.slot[kRho], sX = g.slot[kVxi], sY = g.slot[kVeta], sR = g.slot[kVr], sP = g.slot[kP];
  const T c1 = Coef<T>::drp(1), c2c = Coef<T>::drp(2), c3 = Coef<T>::drp(3);
  const int p2 = (j0 + ty) * n + i0 + V * cx;        // first own point
  // this thread's halo vector: the eta-halo rows first, then the xi-halo columns
  const bool has_halo = tid < NETA + NXI, xi_halo = tid >= NETA;
  int hi, hj;
  if (!xi_halo) {
    const int r = tid / NT;
    hi = (tid % NT) * V;
    hj = r < 3 ? r - 3 : TY + r - 3;
  } else {
    const int q = (tid - NETA) / TY;
    hi = q < QV ? q * V - 4 : TX + (q - QV) * V;
    hj = (tid - NETA) % TY;
  }
  const bool h_in = has_halo && i0 + hi >= 0 && i0 + hi < n && j0 + hj >= 0 && j0 + hj < n;
  const int hq2 = h_in ? (j0 + hj) * n + i0 + hi : 0;
  const int hb = (hj + 3) * PW + hi + 4;             // in a box
  // The 2-D metric terms of the own and of the halo points sit in registers for the chunk.
  T gD[V], gXYD[V], gC[V], gXYC[V], gDivX[V], gDivY[V], gTX[V], gTY[V], gh1[V], gh2[V], gh3[V];
  ldv(a.met + mD * P2 + p2, gD);
  ldv(a.met + mXYD * P2 + p2, gXYD);
  ldv(a.met + mC * P2 + p2, gC);
  ldv(a.met + mXYC * P2 + p2, gXYC);
  ldv(a.met + mDivX * P2 + p2, gDivX);
  ldv(a.met + mDivY * P2 + p2, gDivY);
  ldv(a.met + mTX * P2 + p2, gTX);
  ldv(a.met + mTY * P2 + p2, gTY);
  ldv(a.met + (xi_halo ? mD : mXYD) * P2 + hq2, gh1);
  ldv(a.met + (xi_halo ? mXYC : mC) * P2 + hq2, gh2);
  ldv(a.met + (xi_halo ? mDivX : mDivY) * P2 + hq2, gh3);
  if (tid == 0) {
    for (int q = 0; q < kAdjRing; ++q) mbar_init(&bars[q], 1);
    mbar_fence_init();
  }
  __syncthreads();
  // programmatic launch: everything above reads constant tables only
  grid_dependency_wait();

  // 32-bit offsets inside one face's volumes
  T* const lo_face = a.lout + g.vol(0, face, 0);
  T* const mu_face = a.muout ? a.muout + g.vol(0, face, 0) : nullptr;
  const int vs = (int)g.vs, plane = (int)g.plane;
  const int own0 = (int)g.at(0, j0 + ty, i0 + V * cx);              // own points in plane 0
  const int zf = face * g.nf;            // plane index of (slot s, k) = (zf + s) * nr + k (run 0)
  const int xB = IOFF + i0 - 4, yB = JOFF + j0 - 3, xT = IOFF + i0, yT = JOFF + j0;
  const bool tc2 = a.c2 != nullptr, tdiv = a.grad != nullptr;
  auto slot_base = [&](int sl) { return smem + (size_t)sl * L::SLOT; };
  auto issue = [&](int m, int sl) {
    uint64_t* bar = &bars[sl];
    unsigned char* base = slot_base(sl);
    const int zc = face * nr + m;        // plane index of the compact arrays
    const bool chunk = m >= kb && m < ke;
    uint32_t values = 16;
    if (chunk) values += L::NB * L::PB + L::OB + (a.first ? 0 : L::NF * L::OB) + (tc2 ? L::PB : 0) + (tdiv ? L::OB + L::OB * (sizeof(double) / sizeof(T)) : 0);
    else values += (L::NB - 1 + (tc2 ? 1 : 0)) * L::OB;
    mbar_expect_tx(bar, values * (uint32_t)sizeof(T));
    bulk_load(base + L::RAD, a.radT + (size_t)m * 16, 16 * sizeof(T), bar);
    if (chunk) {
      tma_load_4d(base, &a.mB3, xB, yB, m, zf, bar);
      tma_load_3d(base + L::PBOX, &a.mB, xB, yB, (zf + sP) * nr + m, bar);
      tma_load_3d(base + L::VR, &a.mM, xT, yT, (zf + sR) * nr + m, bar);
      if (!a.first) tma_load_4d(base + L::LQ, &a.mQ, xT, yT, m, zf, bar);
      if (tc2) tma_load_3d(base + L::C2, &a.mC2, i0 - 4, j0 - 3, zc, bar);
      if (tdiv) {
        tma_load_3d(base + L::DIV, &a.mDiv, i0, j0, zc, bar);
        tma_load_3d(base + L::GRAD, &a.mGrad, i0, j0, zc, bar);
      }
    } else {
      tma_load_4d(base, &a.mM2, xT, yT, m, zf + sR, bar);
      if (HAS_RHO) tma_load_3d(base + 2 * L::O_BYTES, &a.mM, xT, yT, (zf + sRho) * nr + m, bar);
      if (tc2) tma_load_3d(base + L::C2, &a.mC2t, i0, j0, zc, bar);
    }
  };
  // planes loaded through the ring: every real plane of [kb-3, ke+2]; planes [m_lo, m_issued)
  // have loads issued, thread 0 has seen planes [m_lo, m_seen) land
  const int m_lo = max(kb - 3, 0), m_hi = min(ke + 2, nr - 1);
  int m_issued = m_lo, m_seen = m_lo;
  const bool loads = !a.wc.no_loads;
  if (tid == 0 && loads) {
    tma_prefetch_desc(&a.mB);
    for (int q = 0; q < kAdjRing && m_issued <= m_hi; ++q, ++m_issued) issue(m_issued, q);
  }
  // facr * dt * (R1, R2) of one of the one-sided rows, from global memory
  auto one_sided = [&](int kk, int row) {
    const T* rr = a.radT + (size_t)kk * 16;
    const T* src = a.mu + g.vol(0, face, 0) + (long long)kk * plane + own0;
    T vp[V], vv[V], vrho[V], cc[V], r1[V], r2[V];
    ldv(src + (long long)sP * vs, vp);
    ldv(src + (long long)sR * vs, vv);
    if (HAS_RHO) ldv(src + (long long)sRho * vs, vrho);
    if (tc2) ldv(a.c2 + ((long long)face * nr + kk) * P2 + p2, cc);
    const T f = a.dt * rr[rFacR], rho0 = rr[rRho0];
#pragma unroll
    for (int q = 0; q < V; ++q) {
      const T c2rho0 = tc2 ? cc[q] * rho0 : rr[rC2Rho0];
      r1[q] = f * (-rr[rInvRho0] * (a.beta * vv[q]));
      r2[q] = -f * (c2rho0 * (a.beta * vp[q]) + (HAS_RHO ? rho0 * (a.beta * vrho[q]) : T(0)));
    }
    T* d = reinterpret_cast<T*>(smem + L::ONE) + (size_t)tid * V;
    stv(d + (2 * row) * L::NTH * V, r1);
    stv(d + (2 * row + 1) * L::NTH * V, r2);
  };
  if (kb <= 6) { one_sided(1, 0); one_sided(2, 1); }

  T ap[7][V], av[7][V];          // partial outputs of p and v_r, planes m-3 .. m+3
  T kp[4][V], kv[4][V];          // alpha * mu of p and v_r, planes m-3 .. m
#pragma unroll
  for (int q = 0; q < V; ++q) {
#pragma unroll
    for (int d = 0; d < 7; ++d) { ap[d][q] = T(0); av[d][q] = T(0); }
#pragma unroll
    for (int d = 0; d < 4; ++d) { kp[d][q] = T(0); kv[d][q] = T(0); }
  }
  T* const held = reinterpret_cast<T*>(smem + L::HELD) + (size_t)tid * V;   // only with LATE
  if constexpr (LATE) stv(held, ap[0]);
  int slot = 0;
  uint32_t phase = 0;
  bool ok = true, failed = false;
  const int bo = (ty + 3) * PW + V * cx + 4;       // own points in a box
  const int to = ty * TX + V * cx;                 // own points in a tile
  const T k2 = -a.dt * a.inv_dxi;
  for (int m = kb - 3; m <= ke + 2; ++m) {
    if (m == ke + 1) release_dependents();
    const bool real = (m >= 0 && m < nr);
    const bool own = (m >= kb && m < ke);
    const bool bc = (m == 0 || m == nr - 1);
    if (real) {
      const int o = m * plane + own0;
      if (ok) {
        ok = mbar_wait(&bars[slot], phase, a.wc, kErrAdjointRing);
        if (ok) m_seen = m + 1;
      }
      const T* sb = reinterpret_cast<const T*>(slot_base(slot));
      const T* sc2 = reinterpret_cast<const T*>(slot_base(slot) + L::C2);
      T rr[12];
#pragma unroll
      for (int q = 0; q < 12; q += V) ldv(reinterpret_cast<const T*>(slot_base(slot) + L::RAD) + q, rr + q);
      const T invr = rr[rInvR], inv_rho0 = rr[rInvRho0], rho0 = rr[rRho0];
      T mP[V], mR[V], mRho[V], cc[V], e[V];        // mu of p, v_r, rho
      ldv(own ? sb + L::PBOX / sizeof(T) + bo : sb + OBs + to, mP);
      ldv(own ? sb + L::VR / sizeof(T) + to : sb + to, mR);
      if (HAS_RHO) ldv(own ? sb + bo : sb + 2 * OBs + to, mRho);
      if (tc2) ldv(own ? sc2 + bo : sc2 + to, cc);
      T lP[V], lR[V], lRho[V];                     // lambda_q (the first stage's boxes hold it)
#pragma unroll
      for (int q = 0; q < V; ++q) {
        lP[q] = mP[q];
        lR[q] = mR[q];
        mP[q] *= a.beta;
        mR[q] *= a.beta;
        if (HAS_RHO) { lRho[q] = mRho[q]; mRho[q] *= a.beta; }
        const T c2rho0 = tc2 ? cc[q] * rho0 : rr[rC2Rho0];
        e[q] = bc ? T(0) : -c2rho0 * mP[q] - (HAS_RHO ? rho0 * mRho[q] : T(0));
      }
      // banded radial transpose (rows 3 .. nr-4): plane m reaches the planes m-3 .. m+3
      if (LATE || (m >= 3 && m <= nr - 4)) {
        const T f = (m >= 3 && m <= nr - 4) ? a.dt * rr[rFacR] : T(0);
        T w1[V], wl[V];                            // of plane m; of plane m-1 where it was held
        if constexpr (LATE) ldv(held, wl);
#pragma unroll
        for (int q = 0; q < V; ++q) w1[q] = f * (-inv_rho0 * mR[q]);
        if constexpr (LATE) stv(held, w1);
#pragma unroll
        for (int q = 0; q < V; ++q) {
          const T w2 = f * e[q];
          ap[0][q] -= c3 * w1[q];
          if constexpr (LATE) ap[1][q] -= c1 * wl[q] + c2c * w1[q];
          else { ap[1][q] -= c2c * w1[q]; ap[2][q] -= c1 * w1[q]; }
          ap[4][q] += c1 * w1[q]; ap[5][q] += c2c * w1[q]; ap[6][q] += c3 * w1[q];
          av[0][q] -= c3 * w2; av[1][q] -= c2c * w2; av[2][q] -= c1 * w2;
          av[4][q] += c1 * w2; av[5][q] += c2c * w2; av[6][q] += c3 * w2;
        }
      }
      if (own) {
        T* const ex = reinterpret_cast<T*>(smem + L::EX + (m & 1) * L::EX_BYTES);
        T* const sX1 = ex;
        T* const sX2 = ex + L::XB;
        T* const sY1 = ex + 2 * L::XB;
        T* const sY2 = ex + 2 * L::XB + L::YB;
        T mX[V], mE[V], lX[V], lE[V];              // v_xi, v_eta
        ldv(sb + R0 * PBs + bo, mX);
        ldv(sb + (R0 + 1) * PBs + bo, mE);
        {
          const T f = -invr * inv_rho0;
          T x1[V], x2[V], y1[V], y2[V];
#pragma unroll
          for (int q = 0; q < V; ++q) {
            lX[q] = mX[q];
            lE[q] = mE[q];
            mX[q] *= a.beta;
            mE[q] *= a.beta;
            const T px = bc ? T(0) : mX[q], pe = bc ? T(0) : mE[q];
            x1[q] = f * (gD[q] * px + gXYC[q] * pe);
            x2[q] = invr * gDivX[q] * e[q];
            y1[q] = f * (gXYD[q] * px + gC[q] * pe);
            y2[q] = invr * gDivY[q] * e[q];
          }
          const int xo = ty * PW + V * cx + 4, yo = (ty + 3) * TX + V * cx;
          stv(sX1 + xo, x1);
          stv(sX2 + xo, x2);
          stv(sY1 + yo, y1);
          stv(sY2 + yo, y2);
        }
        if (has_halo) {
          T v1[V], v2[V];
#pragma unroll
          for (int q = 0; q < V; ++q) { v1[q] = T(0); v2[q] = T(0); }
          if (h_in && !bc) {
            T hx[V], he[V], hp[V], hr[V], hc[V];
            ldv(sb + R0 * PBs + hb, hx);
            ldv(sb + (R0 + 1) * PBs + hb, he);
            ldv(sb + L::PBOX / sizeof(T) + hb, hp);
            if (HAS_RHO) ldv(sb + hb, hr);
            if (tc2) ldv(sc2 + hb, hc);
            const T f = -invr * inv_rho0 * a.beta, fe = -invr * a.beta;
#pragma unroll
            for (int q = 0; q < V; ++q) {
              const T c2rho0 = tc2 ? hc[q] * rho0 : rr[rC2Rho0];
              v1[q] = f * (gh1[q] * hx[q] + gh2[q] * he[q]);
              v2[q] = fe * gh3[q] * (c2rho0 * hp[q] + (HAS_RHO ? rho0 * hr[q] : T(0)));
            }
          }
          const int ho = xi_halo ? hj * PW + hi + 4 : (hj + 3) * TX + hi;
          stv((xi_halo ? sX1 : sY1) + ho, v1);
          stv((xi_halo ? sX2 : sY2) + ho, v2);
        }
        // pointwise terms and the gradient
        if (!a.first) {
          const T* lq = sb + L::LQ / sizeof(T) + to;
          if (HAS_RHO) ldv(lq, lRho);
          ldv(lq + R0 * OBs, lX);
          ldv(lq + (R0 + 1) * OBs, lE);
          ldv(lq + (R0 + 2) * OBs, lR);
          ldv(lq + (R0 + 3) * OBs, lP);
        }
        const T sig = rr[rSigma];
        T orho[V], nrho[V];
        T div[V];
        double gacc[V];
        if (tdiv) {
          ldv(reinterpret_cast<const T*>(slot_base(slot) + L::DIV) + to, div);
#pragma unroll
          for (int q = 0; q < V; q += 2) ldv(reinterpret_cast<const double*>(slot_base(slot) + L::GRAD) + to + q, gacc + q);
        }
#pragma unroll
        for (int q = 0; q < V; ++q) {
          const T pr = bc ? T(0) : mR[q], pp = bc ? T(0) : mP[q];
          T vr_ = T(2) * invr * e[q] + rr[rRho0G0] * pp - sig * mR[q];
          if (HAS_RHO) {
            vr_ -= rr[rDRho0] * (bc ? T(0) : mRho[q]);
            orho[q] = (a.keep ? lRho[q] : T(0)) + a.dt * (-rr[rG0Rho0] * pr - sig * mRho[q]);
            nrho[q] = a.alpha * mRho[q] + a.beta_next * orho[q];
          }
          ap[3][q] -= a.dt * sig * mP[q];
          if constexpr (!LATE) ap[3][q] = (a.keep ? lP[q] : T(0)) + ap[3][q];
          av[3][q] = (a.keep ? lR[q] : T(0)) + (av[3][q] + a.dt * vr_);
          kp[3][q] = a.alpha * mP[q];
          kv[3][q] = a.alpha * mR[q];
          if constexpr (!LATE) {
            lX[q] = (a.keep ? lX[q] : T(0)) - a.dt * (invr * gTX[q] * e[q]);
            lE[q] = (a.keep ? lE[q] : T(0)) - a.dt * (invr * gTY[q] * e[q]);
          }
          if (tdiv) gacc[q] += (double)(a.dt * (rho0 * div[q]) * pp);
        }
        if (tdiv) {
          double* gp = a.grad + ((long long)face * nr + m) * P2 + p2;
#pragma unroll
          for (int q = 0; q < V; q += 2) stv(gp + q, gacc + q);
        }
        if (HAS_RHO) {
          stv(lo_face + sRho * vs + o, orho);
          if (mu_face) stv(mu_face + sRho * vs + o, nrho);
        }
        // every thread is done with the slot and has written its exchange vectors
        fence_reads_before_copies();
        if (__syncthreads_or(!ok)) { failed = true; break; }
        if (tid == 0 && loads && m_issued <= m_hi) issue(m_issued++, slot);
        T w1[NV * V], w2[NV * V];
#pragma unroll
        for (int q = 0; q < NV; ++q) {
          ldv(sX1 + ty * PW + (cx + q) * V, w1 + q * V);
          ldv(sX2 + ty * PW + (cx + q) * V, w2 + q * V);
        }
        T d1[V], d2[V], dy2[V];
        {
          T u[3][V], d[3][V];
          const int yo = (ty + 3) * TX + V * cx;
#pragma unroll
          for (int r = 1; r <= 3; ++r) { ldv(sY1 + yo + r * TX, u[r - 1]); ldv(sY1 + yo - r * TX, d[r - 1]); }
#pragma unroll
          for (int q = 0; q < V; ++q)
            d1[q] = c1 * (u[0][q] - d[0][q]) + c2c * (u[1][q] - d[1][q]) + c3 * (u[2][q] - d[2][q]);
#pragma unroll
          for (int r = 1; r <= 3; ++r) { ldv(sY2 + yo + r * TX, u[r - 1]); ldv(sY2 + yo - r * TX, d[r - 1]); }
#pragma unroll
          for (int q = 0; q < V; ++q)
            dy2[q] = c1 * (u[0][q] - d[0][q]) + c2c * (u[1][q] - d[1][q]) + c3 * (u[2][q] - d[2][q]);
        }
        auto dxi = [&](const T* w, int c) {        // c = index into the window; zero past it
          auto at = [&](int q) { return (q >= 0 && q < NV * V) ? w[q] : T(0); };
          return c1 * (at(c + 1) - at(c - 1)) + c2c * (at(c + 2) - at(c - 2)) + c3 * (at(c + 3) - at(c - 3));
        };
        T nX[V], nE[V];
#pragma unroll
        for (int q = 0; q < V; ++q) {
          d1[q] += dxi(w1, 4 + q);
          d2[q] = dxi(w2, 4 + q);
          if constexpr (LATE) {
            ap[3][q] = (a.keep ? lP[q] : T(0)) + (ap[3][q] + k2 * d1[q]);
            lX[q] = (a.keep ? lX[q] : T(0)) + (k2 * d2[q] - a.dt * (invr * gTX[q] * e[q]));
            lE[q] = (a.keep ? lE[q] : T(0)) + (k2 * dy2[q] - a.dt * (invr * gTY[q] * e[q]));
          } else {
            ap[3][q] += k2 * d1[q];
            lX[q] += k2 * d2[q];
            lE[q] += k2 * dy2[q];
          }
          nX[q] = a.alpha * mX[q] + a.beta_next * lX[q];
          nE[q] = a.alpha * mE[q] + a.beta_next * lE[q];
        }
        stv(lo_face + sX * vs + o, lX);
        stv(lo_face + sY * vs + o, lE);
        if (mu_face) {
          stv(mu_face + sX * vs + o, nX);
          stv(mu_face + sY * vs + o, nE);
        }
        // ghost-frame adjoints of the neighbour faces' values (W/E columns, S/N rows); the
        // exchange arrays are zero outside the face
        if (i0 == 0 && cx == 0) {
#pragma unroll
          for (int c = 1; c <= 3; ++c) {
            lo_face[sP * vs + o - 4 + c] = k2 * dxi(w1, c);
            lo_face[sX * vs + o - 4 + c] = k2 * dxi(w2, c);
          }
        }
        if (i0 + TX == n && cx == NT - 1) {
#pragma unroll
          for (int c = V + 4; c <= V + 6; ++c) {
            lo_face[sP * vs + o - 4 + c] = k2 * dxi(w1, c);
            lo_face[sX * vs + o - 4 + c] = k2 * dxi(w2, c);
          }
        }
        const bool south = j0 == 0 && ty < 3, north = j0 + TY == n && ty >= TY - 3;
        if (south || north) {
#pragma unroll
          for (int side = 0; side < 2; ++side) {
            if (side == 0 ? !south : !north) continue;
            const int r = side == 0 ? ty : ty + 6;           // exchange row of the ghost row
            auto dy = [&](const T* y, int q) {
              auto at = [&](int row) { return (row >= 0 && row < YH) ? y[row * TX + V * cx + q] : T(0); };
              return c1 * (at(r + 1) - at(r - 1)) + c2c * (at(r + 2) - at(r - 2)) + c3 * (at(r + 3) - at(r - 3));
            };
            T f1[V], f2[V];
#pragma unroll
            for (int q = 0; q < V; ++q) { f1[q] = k2 * dy(sY1, q); f2[q] = k2 * dy(sY2, q); }
            const int og = o + (side == 0 ? -3 : 3) * g.pitch;
            stv(lo_face + sP * vs + og, f1);
            stv(lo_face + sY * vs + og, f2);
          }
        }
      } else {
        fence_reads_before_copies();
        if (__syncthreads_or(!ok)) { failed = true; break; }
        if (tid == 0 && loads && m_issued <= m_hi) issue(m_issued++, slot);
      }
      if (++slot == kAdjRing) { slot = 0; phase ^= 1; }
    } else if constexpr (LATE) {                   // beside the shell: only the held term
      T wl[V];
      ldv(held, wl);
#pragma unroll
      for (int q = 0; q < V; ++q) {
        ap[1][q] -= c1 * wl[q];
        wl[q] = T(0);
      }
      stv(held, wl);
    }
    const int pl = m - 3;
    if (pl >= kb && pl < ke) {
      if (pl < 7 || pl >= nr - 7) {
        const bool low = pl < 7;
        if (!low && pl == max(kb, nr - 7)) { one_sided(nr - 3, 0); one_sided(nr - 2, 1); }
        const T* d = reinterpret_cast<const T*>(smem + L::ONE) + (size_t)tid * V;
        T s1[V], s2[V];
#pragma unroll
        for (int row = 0; row < 2; ++row) {
          const T b = low ? Coef<T>::bdy(1 + row, pl) : -Coef<T>::bdy(2 - row, nr - 1 - pl);
          T r1[V], r2[V];
          ldv(d + (2 * row) * L::NTH * V, r1);
          ldv(d + (2 * row + 1) * L::NTH * V, r2);
#pragma unroll
          for (int q = 0; q < V; ++q) {
            s1[q] = row ? s1[q] + b * r1[q] : b * r1[q];
            s2[q] = row ? s2[q] + b * r2[q] : b * r2[q];
          }
        }
#pragma unroll
        for (int q = 0; q < V; ++q) { ap[0][q] += s1[q]; av[0][q] += s2[q]; }
      }
      const int op = pl * plane + own0;
      stv(lo_face + sP * vs + op, ap[0]);
      stv(lo_face + sR * vs + op, av[0]);
      if (mu_face) {
#pragma unroll
        for (int q = 0; q < V; ++q) {
          kp[0][q] += a.beta_next * ap[0][q];
          kv[0][q] += a.beta_next * av[0][q];
        }
        stv(mu_face + sP * vs + op, kp[0]);
        stv(mu_face + sR * vs + op, kv[0]);
      }
    }
    // the partial outputs advance one plane
#pragma unroll
    for (int q = 0; q < V; ++q) {
#pragma unroll
      for (int d = 0; d < 6; ++d) { ap[d][q] = ap[d + 1][q]; av[d][q] = av[d + 1][q]; }
      ap[6][q] = T(0);
      av[6][q] = T(0);
#pragma unroll
      for (int d = 0; d < 3; ++d) { kp[d][q] = kp[d + 1][q]; kv[d][q] = kv[d + 1][q]; }
      kp[3][q] = T(0);
      kv[3][q] = T(0);
    }
  }
  // a wait gave up: wait (bounded) for the loads still in flight before the CTA exits
  if (failed && tid == 0 && loads) mbar_drain(bars, kAdjRing, m_lo, m_seen, m_issued, a.wc.polls);
}

// The gradient's last factor: grad holds sum dt rho0 div mu_p; dJ/dc = -2 c times that.
template <typename T>
__global__ void grad_scale_kernel(double* grad, const T* c2, const T* radT, int nr, long long P2) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= 6 * nr * P2) return;
  const T* rr = radT + (size_t)((idx / P2) % nr) * 16;
  const T c = sqrt(c2 ? c2[idx] : rr[rC2Rho0] * rr[rInvRho0]);
  grad[idx] = -2.0 * (double)c * grad[idx];
}

// Transpose of the edge exchange, as a gather: every source-line point (the receiving face
// and edge's route, layer l, position u along the source edge, plane k) sums the ghost
// adjoints of the ghost points whose 9 taps include it -- a contiguous range of positions t,
// tspan -- then adds the sum to its value (atomically: the source lines of two edges of a
// face share their corner points).  The CTA first copies the ghost values its positions
// need (the union of their ranges, one read per ghost point and field) into shared memory:
// on W/E receivers those are column entries, one scattered request each.  The weights come
// from a table transposed on the host, wt[kind][row][j][u] = the folded coefficient with
// which ghost point t = lo(u) + j of row (face-edge, layer) used source position u (kind 0
// scalar, 1 and 2 the vector pair), read contiguously across u.  mode 0: p scalar + the
// rotated vector component (v_xi on W/E receivers, v_eta on S/N); mode 1: every stored
// field scalar.  grid: x over u, y over (receiving face-edge, layer), z over planes; dynamic
// shared memory: (mode 0 ? 2 : nf) x n values.
template <typename T>
struct AdjEdgeArgs {
  T* q;
  T* mu;                  // or nullptr
  T beta;
  const T* wt;
  int span;
  const int* tspan;
  Geom g;
  int mode;
};

template <typename T>
__global__ void adj_edge_kernel(const __grid_constant__ AdjEdgeArgs<T> a) {
  T* const q = a.q;
  T* const mu = a.mu;
  const T beta = a.beta;
  const T* __restrict__ wt = a.wt;
  const int* __restrict__ tspan = a.tspan;
  const int span = a.span, mode = a.mode;
  const Geom& g = a.g;
  extern __shared__ __align__(16) unsigned char aesm[];
  T* const sg = reinterpret_cast<T*>(aesm);               // [field][t]
  __shared__ int s_lo, s_hi;
  const int n = g.n;
  const int u = blockIdx.x * blockDim.x + threadIdx.x;
  const int fe = blockIdx.y / 3, l = blockIdx.y % 3, k = blockIdx.z;
  const int face = fe >> 2, e = fe & 3;
  const EdgeRouteDev rt = cRoute[face][e];
  const bool along_i = rt.src_edge <= 1;
  const int fixed = (rt.src_edge == 0 || rt.src_edge == 2) ? l + 1 : n - 2 - l;
  const int row = fe * 3 + l;
  int lo = 0, hi = -1;
  if (u < n) {
    lo = __ldg(tspan + (row * n + u) * 2);
    hi = __ldg(tspan + (row * n + u) * 2 + 1);
  }
  if (threadIdx.x == 0) { s_lo = n; s_hi = -1; }
  __syncthreads();
  if (hi >= lo) { atomicMin(&s_lo, lo); atomicMax(&s_hi, hi); }
  __syncthreads();
  const int tmin = s_lo, tmax = s_hi;
  grid_dependency_wait();                                  // constant tables only above
  release_dependents();
  if (tmax < tmin) return;                                 // no ghost point uses this block
  // receiver ghost position of (e, l, t): rows -1-l / n+l, columns -1-l / n+l
  const long long g0 = (e == 0) ? g.at(k, -1 - l, 0) : (e == 1) ? g.at(k, n + l, 0)
                     : (e == 2) ? g.at(k, 0, -1 - l) : g.at(k, 0, n + l);
  const long long gstep = e <= 1 ? 1 : g.pitch;
  const int nfs = mode == 1 ? g.nf : 2;
  auto slot_of = [&](int f) {
    return mode == 1 ? f : (f == 0 ? g.slot[kP] : (e >= 2 ? g.slot[kVxi] : g.slot[kVeta]));
  };
  for (int f = 0; f < nfs; ++f) {
    const T* gv = q + g.vol(0, face, slot_of(f)) + g0;
    for (int t = tmin + threadIdx.x; t <= tmax; t += blockDim.x) sg[f * n + t] = gv[t * gstep];
  }
  __syncthreads();
  if (hi < lo) return;
  const long long src = g.at(k, along_i ? fixed : u, along_i ? u : fixed);
  const long long kind = 72LL * span * n;                 // stride between weight kinds
  const T* w = wt + (long long)row * span * n + u;        // weight of ghost lo + j at w[j * n]
  const int cnt = hi - lo + 1;
  if (mode == 1) {
    for (int f = 0; f < nfs; ++f) {
      const T* gs = sg + f * n + lo;
      T acc = T(0);
      for (int j = 0; j < cnt; ++j) acc += __ldg(w + j * n) * gs[j];
      atomicAdd(q + g.vol(0, rt.src_face, f) + src, acc);
    }
    return;
  }
  const T* gp = sg + lo;
  const T* gvv = sg + n + lo;
  T ap = T(0), ax = T(0), ay = T(0);
  for (int j = 0; j < cnt; ++j) {
    const T pv = gp[j], vv = gvv[j];
    ap += __ldg(w + j * n) * pv;
    ax += __ldg(w + kind + j * n) * vv;
    ay += __ldg(w + 2 * kind + j * n) * vv;
  }
  const long long op = g.vol(0, rt.src_face, g.slot[kP]) + src, ox = g.vol(0, rt.src_face, g.slot[kVxi]) + src,
                  oy = g.vol(0, rt.src_face, g.slot[kVeta]) + src;
  atomicAdd(q + op, ap);
  atomicAdd(q + ox, ax);
  atomicAdd(q + oy, ay);
  if (mu) {                                               // mu = alpha mu + beta lambda_q
    atomicAdd(mu + op, beta * ap);
    atomicAdd(mu + ox, beta * ax);
    atomicAdd(mu + oy, beta * ay);
  }
}

// FILTER_EXP^T of one field on the face interior, fused.  The transpose is radial^T, then eta^T,
// then xi^T; the three act along different axes, so they commute and the radial one can come
// last, on a register queue as in filter_kernel: per plane the xi and eta filters with zero
// halos (the tensor map covers the interior only, so the load fills them), then the 11-point
// radial filter over the planes [5, nr-6] (the forward output is zero outside them).  Every sum runs
// from the outer taps to the centre: the rounding of a sum counts where it is large, and the radial
// filter, being last, is followed by none that smooths it (error in float 4.8e-8; centre first
// 8.4e-8, with the radial filter first and the xi filter last 7.5e-8; the same time).  Tiles,
// threads, ring and work split are those of filter_kernel, and so is what bounds it.  us per
// launch at 6 x 96^3 in double / float: 117 / 55, and adj_ghost_kernel 42 / 29 after it (as a
// radial pass over the whole buffer and a plane-marching xi/eta pass with plain loads, ghost
// adjoints included, 117 + 170 / 52 + 67; with a branch around the zero planes 134 / 69).
template <typename T, int TX, int TY, int R>
__global__ void __launch_bounds__((TX / Vec16<T>::V) * (TY / R), sizeof(T) == 4 ? 4 : 1) adj_filter_kernel(const __grid_constant__ FilterArgs<T> a) {
  constexpr int V = Vec16<T>::V, NT = TX / V, NY = TY / R, NV = (V + 8) / V, PW = TX + 8, NP = V / 2;
  constexpr bool PAIRS = sizeof(T) == 4;
  using L = FilterLayout<T, TX, TY>;
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR);
  const Geom& g = a.g;
  const int n = g.n, nr = g.nr;
  const int tiles_x = n / TX, tiles = tiles_x * (n / TY);
  int unit = blockIdx.x, ko0 = 0, ko1 = nr;
  if (unit >= a.whole) {
    const int t = unit - a.whole, c = t % a.chunks;
    unit = a.whole + t / a.chunks;
    ko0 = c * nr / a.chunks;
    ko1 = (c + 1) * nr / a.chunks;
  }
  const int ks = ko0 - 5, ke = ko1 + 5;                        // input planes, zero outside [5, nr-6]
  const int tile = unit % tiles, rest = unit / tiles;
  const int i0 = (tile % tiles_x) * TX, j0 = (tile / tiles_x) * TY;
  const int s = rest % g.nf, face = rest / g.nf;
  const int cx = threadIdx.x, ty = threadIdx.y, tid = ty * NT + cx;
  const int rb = R * ty;                     // first own row of the tile
  const int z0 = (face * g.nf + s) * nr;
  auto issue = [&](int k, int slot) {
    uint64_t* b = &bars[slot];
    mbar_expect_tx(b, L::PB * sizeof(T));
    const bool in = k >= 5 && k < nr - 5;              // else a box beside the face, all zeros
    tma_load_3d(smem + slot * L::P_BYTES, &a.mP, in ? i0 - 4 : n, j0 - 3, z0 + (in ? k : 5), b);
  };
  if (tid == 0) {
    for (int q = 0; q < kFiltRing; ++q) mbar_init(&bars[q], 1);
    mbar_fence_init();
  }
  __syncthreads();
  grid_dependency_wait();
  const bool loads = !a.wc.no_loads;
  if (tid == 0 && loads)
    for (int k = ks; k < min(ks + kFiltRing, ke); ++k) issue(k, k - ks);
  T* out = a.qout + g.vol(0, face, s) + g.at(0, j0 + rb, i0 + V * cx);
  constexpr T f0 = T(kFilt[0]), f1 = T(kFilt[1]), f2 = T(kFilt[2]), f3 = T(kFilt[3]);
  constexpr T rw[6] = {T(kFiltR[0]), T(kFiltR[1]), T(kFiltR[2]), T(kFiltR[3]), T(kFiltR[4]), T(kFiltR[5])};
  auto xi_row = [&](const T* bx, int r, T* v) {       // xi filter of box row r at the own columns
    T w[NV * V];
#pragma unroll
    for (int m = 0; m < NV; ++m) ldv(bx + r * PW + V * cx + m * V, w + m * V);
#pragma unroll
    for (int q = 0; q < V; ++q)
      v[q] = f3 * (w[1 + q] + w[7 + q]) + f2 * (w[2 + q] + w[6 + q]) + f1 * (w[3 + q] + w[5 + q]) + f0 * w[4 + q];
  };
  // radial queue of eta-filtered planes, in float as packed pairs (filter_kernel)
  T tq[11][R][V];
  unsigned long long tq2[11][R][NP];
#pragma unroll
  for (int m = 0; m < 11; ++m)
#pragma unroll
    for (int r = 0; r < R; ++r) {
#pragma unroll
      for (int q = 0; q < V; ++q) tq[m][r][q] = T(0);
#pragma unroll
      for (int h = 0; h < NP; ++h) tq2[m][r][h] = 0ull;
    }
  // A thread whose wait gives up reports it at the CTA barrier; the CTA leaves the plane loop
  // there (fail_at = 2 * plane + whether thread 0's own wait on that plane succeeded).
  bool ok = true;
  int fail_at = 0;
  int slot = 0;
  uint32_t phase = 0;
  for (int kb = ks; kb < ke && ok; kb += 11) {
#pragma unroll
    for (int u = 0; u < 11; ++u) {
      const int k = kb + u;
      if (k >= ke) break;
      if (k == ke - release_planes(ke - ks)) release_dependents();
      {
        const bool got = mbar_wait(&bars[slot], phase, a.wc, kErrAdjointFilter);
        const T* bx = reinterpret_cast<const T*>(smem + slot * L::P_BYTES);
        T* t1 = reinterpret_cast<T*>(smem + kFiltRing * L::P_BYTES + (k & 1) * L::S_BYTES);
        T c[R + 6][V];                                 // c[m] holds xi-filtered box row rb + m
#pragma unroll
        for (int r = 0; r < R; ++r) {
          xi_row(bx, rb + 3 + r, c[3 + r]);
          stv(t1 + (rb + 3 + r) * TX + V * cx, c[3 + r]);
        }
        for (int h = ty; h < 6; h += NY) {             // the halo rows of the box
          const int r = h < 3 ? h : TY + h;
          T v[V];
          xi_row(bx, r, v);
          stv(t1 + r * TX + V * cx, v);
        }
        if (__syncthreads_or(!got)) { ok = false; fail_at = 2 * k + (got ? 1 : 0); break; }
        if (tid == 0 && loads && k + kFiltRing < ke) issue(k + kFiltRing, slot);
        if (++slot == kFiltRing) { slot = 0; phase ^= 1; }
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          ldv(t1 + (rb + m) * TX + V * cx, c[m]);
          ldv(t1 + (rb + R + 3 + m) * TX + V * cx, c[R + 3 + m]);
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
          if constexpr (PAIRS) {
#pragma unroll
            for (int h = 0; h < NP; ++h) {
              auto pr = [&](int m) { return pk2(c[r + m][2 * h], c[r + m][2 * h + 1]); };
              unsigned long long t = mul2(pk2(f3, f3), add2(pr(0), pr(6)));
              t = fma2(pk2(f2, f2), add2(pr(1), pr(5)), t);
              t = fma2(pk2(f1, f1), add2(pr(2), pr(4)), t);
              tq2[u][r][h] = fma2(pk2(f0, f0), pr(3), t);
            }
          } else {
#pragma unroll
            for (int q = 0; q < V; ++q)
              tq[u][r][q] = f3 * (c[r][q] + c[r + 6][q]) + f2 * (c[r + 1][q] + c[r + 5][q]) +
                            f1 * (c[r + 2][q] + c[r + 4][q]) + f0 * c[r + 3][q];
          }
        }
      }
      if (k >= ko0 + 5) {
        // planes k-10 .. k sit at queue rows (u+1 .. u+11) % 11; the centre is k-5
#pragma unroll
        for (int r = 0; r < R; ++r) {
          T v[V];
          if constexpr (PAIRS) {
#pragma unroll
            for (int h = 0; h < NP; ++h) {
              unsigned long long acc = mul2(pk2(rw[5], rw[5]), add2(tq2[(u + 1) % 11][r][h], tq2[(u + 11) % 11][r][h]));
#pragma unroll
              for (int m = 4; m >= 1; --m)
                acc = fma2(pk2(rw[m], rw[m]), add2(tq2[(u + 6 - m) % 11][r][h], tq2[(u + 6 + m) % 11][r][h]), acc);
              float x, y;
              upk2(fma2(pk2(rw[0], rw[0]), tq2[(u + 6) % 11][r][h], acc), x, y);
              v[2 * h] = x;
              v[2 * h + 1] = y;
            }
          } else {
#pragma unroll
            for (int q = 0; q < V; ++q) {
              T acc = rw[5] * (tq[(u + 1) % 11][r][q] + tq[(u + 11) % 11][r][q]);
#pragma unroll
              for (int m = 4; m >= 1; --m) acc += rw[m] * (tq[(u + 6 - m) % 11][r][q] + tq[(u + 6 + m) % 11][r][q]);
              v[q] = acc + rw[0] * tq[(u + 6) % 11][r][q];
            }
          }
          stv(out + (long long)(k - 5) * g.plane + r * g.pitch, v);
        }
      }
    }
  }
  if (!ok && tid == 0 && loads) {
    // at the break on plane k, planes [ks, min(k + kFiltRing, ke)) were issued
    const int k = fail_at >> 1;
    mbar_drain(bars, kFiltRing, ks, k + (fail_at & 1), min(k + kFiltRing, ke), a.wc.polls);
  }
}

// Ghost adjoints of FILTER_EXP^T, from the interior of `in` into the frame of `out`.  The eta
// filter's halo took the unfiltered rows, so the ghost rows are the eta transpose of u alone,
// sums of the three rows next to the edge; the ghost columns are the xi transpose of eta^T u,
// sums of the three columns next to it.  Both are then filtered radially, with an 11-deep
// register queue of the three values per thread, over a chunk of kp planes.  grid.z: volume and
// edge.  Ghost rows: one thread per column.  Ghost columns: one lane per row, which reads the
// aligned group of four values once per plane and takes its neighbours' from the other lanes
// (lanes 3..28 write); reading 7 rows per thread, or one layer per thread, is bound by the
// scattered requests.
template <typename T>
struct AdjGhostArgs {
  const T* in;
  T* out;
  Geom g;
  int kp;
};

template <typename T>
__global__ void __launch_bounds__(128) adj_ghost_kernel(const __grid_constant__ AdjGhostArgs<T> a) {
  const Geom& g = a.g;
  const int n = g.n, nr = g.nr;
  const int e = blockIdx.z & 3;
  const T* in = a.in + (long long)(blockIdx.z >> 2) * g.vs;
  T* out = a.out + (long long)(blockIdx.z >> 2) * g.vs;
  const int k0 = blockIdx.y * a.kp, k1 = min(nr, k0 + a.kp);
  constexpr T f0 = T(kFilt[0]), f1 = T(kFilt[1]), f2 = T(kFilt[2]), f3 = T(kFilt[3]);
  constexpr T rw[6] = {T(kFiltR[0]), T(kFiltR[1]), T(kFiltR[2]), T(kFiltR[3]), T(kFiltR[4]), T(kFiltR[5])};
  const bool cols = e >= 2;
  const int lane = threadIdx.x & 31, gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int t = cols ? gw * 26 + lane - 3 : (int)(blockIdx.x * blockDim.x + threadIdx.x);   // row or column
  const bool in_face = t >= 0 && t < n, writes = in_face && (!cols || (lane >= 3 && lane < 29));
  grid_dependency_wait();
  release_dependents();
  if (cols ? gw * 26 >= n : t >= n) return;                  // whole warps (columns) or lone threads
  // the three values next to the edge of plane k, nearest first (eta-filtered for the columns)
  auto load = [&](int k, T* v) {
    v[0] = v[1] = v[2] = T(0);
    if (k < 5 || k > nr - 6) return;                         // uniform over the grid's block row
    if (!cols) {
#pragma unroll
      for (int l = 0; l < 3; ++l) v[l] = in[g.at(k, e == 0 ? l : n - 1 - l, t)];
      return;
    }
    T u[4] = {T(0), T(0), T(0), T(0)};
    if (in_face) {
      const T* p = in + g.at(k, t, e == 2 ? 0 : n - 4);
      ldv(p, u);
      if (sizeof(T) == 8) ldv(p + 2, u + 2);
    }
#pragma unroll
    for (int l = 0; l < 3; ++l) {
      const T x = e == 2 ? u[l] : u[3 - l];
      T s = f3 * (__shfl_up_sync(0xffffffffu, x, 3) + __shfl_down_sync(0xffffffffu, x, 3));
      s += f2 * (__shfl_up_sync(0xffffffffu, x, 2) + __shfl_down_sync(0xffffffffu, x, 2));
      s += f1 * (__shfl_up_sync(0xffffffffu, x, 1) + __shfl_down_sync(0xffffffffu, x, 1));
      v[l] = s + f0 * x;
    }
  };
  T q[11][3];
#pragma unroll
  for (int d = 0; d < 11; ++d) load(k0 + d - 5, q[d]);       // planes m-5 .. m+5 for m = k0
  for (int m = k0; m < k1; ++m) {
    T s[3];
#pragma unroll
    for (int l = 0; l < 3; ++l) {
      s[l] = rw[5] * (q[0][l] + q[10][l]);
#pragma unroll
      for (int d = 4; d >= 1; --d) s[l] += rw[d] * (q[5 - d][l] + q[5 + d][l]);
      s[l] += rw[0] * q[5][l];
    }
    const T w[3] = {f1 * s[0] + f2 * s[1] + f3 * s[2], f2 * s[0] + f3 * s[1], f3 * s[0]};   // layers 1, 2, 3
    if (writes) {
      if (!cols) {
#pragma unroll
        for (int l = 0; l < 3; ++l) out[g.at(m, e == 0 ? -1 - l : n + l, t)] = w[l];
      } else {                                               // the group of four: columns -4..-1 or n..n+3
        T v[4];
#pragma unroll
        for (int l = 0; l < 3; ++l) v[e == 2 ? 3 - l : l] = w[l];
        v[e == 2 ? 0 : 3] = T(0);
        T* p = out + g.at(m, t, e == 2 ? -4 : n);
        stv(p, v);
        if (sizeof(T) == 8) stv(p + 2, v + 2);
      }
    }
#pragma unroll
    for (int d = 0; d < 10; ++d)
#pragma unroll
      for (int l = 0; l < 3; ++l) q[d][l] = q[d + 1][l];
    load(m + 6, q[10]);
  }
}

// Receivers: p sampled with trilinear weights over the 8 grid points around each receiver
// on its face.  rec_off[r*8+c] is the padded-buffer offset of corner c (p slot, run 0) and
// rec_w[r*8+c] its weight.  inject_kernel is the transpose of sample_kernel.
template <typename T>
__global__ void sample_kernel(const T* q, const long long* rec_off, const double* rec_w, int nrec, double* out) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nrec) return;
  double s = 0.0;
  for (int c = 0; c < 8; ++c) s += rec_w[r * 8 + c] * (double)q[rec_off[r * 8 + c]];
  out[r] = s;
}

template <typename T>
__global__ void inject_kernel(T* lam, const long long* rec_off, const double* rec_w, int nrec, const double* res) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nrec) return;
  for (int c = 0; c < 8; ++c) atomicAdd(lam + rec_off[r * 8 + c], (T)(rec_w[r * 8 + c] * res[r]));
}

}  // namespace solar
