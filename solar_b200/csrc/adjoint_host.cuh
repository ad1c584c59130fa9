// adjoint_host.cuh -- host side of the discrete adjoint: receivers, checkpointed reverse
// sweep and the C-ABI entry points declared in include/solar_gpu.h.  Included once, by
// solar_gpu.cu: the adjoint kernels read the scheme constants that live in that
// translation unit's constant memory.
#pragma once

#include "adjoint.cuh"

namespace solar {

static long long state_bytes(const solar_ctx* c) { return 6LL * c->g.nf * c->g.vs * (long long)c->esize; }

static int adj_alloc(solar_ctx* c) {
  AdjBuffers& b = c->adj;
  if (c->g.nface != 6) return fail(SOLAR_ERR_ARG, "the adjoint entry points need a context owning all six zones");
  if (b.L) return SOLAR_OK;
  if (c->g.nruns != 1) return fail(SOLAR_ERR_ARG, "the adjoint entry points need nruns == 1");
  const size_t S = (size_t)state_bytes(c);
  void** bufs[4] = {&b.L, &b.LW, &b.T1, &b.T2};
  for (void** p : bufs) {
    if (cudaMalloc(p, S) != cudaSuccess) { cudaGetLastError(); return fail(SOLAR_ERR_NOMEM, "adjoint buffers: out of device memory"); }
    CK(cudaMemsetAsync(*p, 0, S, c->stream));
  }
  CK(cudaMalloc((void**)&b.grad, (size_t)6 * vol_compact(c) * sizeof(double)));
  CK(cudaMalloc((void**)&b.tspan, c->ht.tspan.size() * sizeof(int)));
  CK(cudaMemcpy(b.tspan, c->ht.tspan.data(), c->ht.tspan.size() * sizeof(int), cudaMemcpyHostToDevice));
  // Edge weights transposed to the gather's order: wt[kind][row][j][u] is the coefficient
  // with which ghost point t = lo(u) + j of row (face-edge, layer) used source position u
  // (kind 0: scalar weight, 1 and 2: the vector pair); zero past the ghost range of u.
  const int n = c->g.n;
  int span = 1;
  for (size_t q = 0; q < c->ht.tspan.size(); q += 2) span = std::max(span, c->ht.tspan[q + 1] - c->ht.tspan[q] + 1);
  std::vector<double> wt((size_t)3 * 72 * span * n, 0.0);
  for (int row = 0; row < 72; ++row)
    for (int u = 0; u < n; ++u) {
      const int lo = c->ht.tspan[((size_t)row * n + u) * 2], hi = c->ht.tspan[((size_t)row * n + u) * 2 + 1];
      for (int t = lo; t <= hi; ++t) {
        const int s = u - c->ht.s0t[(size_t)row * n + t];
        if (s < 0 || s > 8) continue;
        const size_t tap = (size_t)row * 9 + s, o = ((size_t)row * span + (t - lo)) * n + u;
        wt[o] = c->ht.ew[tap * n + t];
        wt[(size_t)72 * span * n + o] = c->ht.eg[(tap * 2 + 0) * n + t];
        wt[(size_t)2 * 72 * span * n + o] = c->ht.eg[(tap * 2 + 1) * n + t];
      }
    }
  int rc = c->fp32 ? upload<float>(&b.wt, wt) : upload<double>(&b.wt, wt);
  if (rc) return rc;
  b.wt_span = span;
  return SOLAR_OK;
}

// Grow-only device arrays of the adjoint (checkpoints, stage divergences, traces).
static int adj_reserve(void** p, size_t* have, size_t want) {
  if (*have >= want) return SOLAR_OK;
  if (*p) cudaFree(*p);
  *p = nullptr;
  *have = 0;
  if (cudaMalloc(p, want) != cudaSuccess) {
    cudaGetLastError();
    return fail(SOLAR_ERR_NOMEM, "adjoint: cannot allocate %.2f GB of device memory", want / 1e9);
  }
  *have = want;
  return SOLAR_OK;
}

// Arguments of one transposed stage; as they stand, out = dt L^T(L) without the RK recursion.
template <typename T>
static AdjStageArgs<T> adj_args(solar_ctx* c, double dt) {
  AdjStageArgs<T> a = {};
  a.c2 = (const T*)c->dt.c2;
  a.met = (const T*)c->dt.met;
  a.radT = (const T*)c->dt.radT;
  a.g = c->g;
  a.beta = T(1);
  a.dt = (T)dt;
  a.inv_dxi = (T)(1.0 / c->ht.dxi);
  a.first = 1;
  a.wc = wait_ctl(c, kInjAdjStage);
  return a;
}

static unsigned blocks_for(long long n, int threads) { return (unsigned)((n + threads - 1) / threads); }

template <typename T, int TX, int TY, bool HAS_RHO>
static int launch_adj_stage_t(solar_ctx* c, AdjStageArgs<T>& a) {
  using L = AdjLayout<T, TX, TY, HAS_RHO>;
  AdjBuffers& b = c->adj;
  if (!make_fields_map(c, a.mu, TX + 8, TY + 6, HAS_RHO ? 3 : 2, &a.mB3) || !make_map(c, a.mu, TX + 8, TY + 6, &a.mB) ||
      !make_map(c, a.mu, TX, TY, &a.mM) || !make_fields_map(c, a.mu, TX, TY, 2, &a.mM2) ||
      !make_fields_map(c, b.L, TX, TY, c->g.nf, &a.mQ) ||
      (a.c2 && (!make_compact_map(c, a.c2, TX + 8, TY + 6, &a.mC2) || !make_compact_map(c, a.c2, TX, TY, &a.mC2t))) ||
      (a.grad && (!make_compact_map(c, a.div, TX, TY, &a.mDiv) || !make_compact_map(c, a.grad, TX, TY, &a.mGrad, true))))
    return fail(SOLAR_ERR_CUDA, "cuTensorMapEncodeTiled failed");
  if (!a.c2) a.mC2 = a.mC2t = a.mM;               // unused
  if (!a.grad) a.mDiv = a.mGrad = a.mM;
  static bool attr_set = false;
  static int resident = 1;
  if (!attr_set) {
    CK(cudaFuncSetAttribute(adj_stage_kernel<T, TX, TY, HAS_RHO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::TOTAL));
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, adj_stage_kernel<T, TX, TY, HAS_RHO>, L::NTH, L::TOTAL));
    resident = std::max(resident, 1);
    attr_set = true;
  }
  const Geom& g = c->g;
  // Radial chunks: the count that minimises waves x (planes per CTA + 3): the three extra planes
  // on either side move few bytes (us per reverse step at 6 x 96^3, float: + 3 850, + 6 862, + 9
  // 1004; the same within 0.2% in double).
  const long long tiles = 6LL * (g.n / TX) * (g.n / TY);
  const long long slots = (long long)c->nsm * resident;
  int best = 1;
  long long best_cost = -1;
  for (int nch = 1; nch <= g.nr; ++nch) {
    const long long kc = (g.nr + nch - 1) / nch;
    const long long cost = ((tiles * nch + slots - 1) / slots) * (kc + 3);
    if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = nch; }
  }
  a.kchunk = (g.nr + best - 1) / best;
  dim3 grid((unsigned)((g.n / TX) * (g.n / TY)), (unsigned)((g.nr + a.kchunk - 1) / a.kchunk), 6);
  CK(launch_pdl(adj_stage_kernel<T, TX, TY, HAS_RHO>, grid, dim3(TX / L::V, TY), L::TOTAL, c->stream, a));
  return SOLAR_OK;
}

template <typename T, int TX, int TY>
static int launch_adj_stage(solar_ctx* c, AdjStageArgs<T>& a) {
  return c->g.slot[kRho] >= 0 ? launch_adj_stage_t<T, TX, TY, true>(c, a) : launch_adj_stage_t<T, TX, TY, false>(c, a);
}

// One transposed stage on the buffers L (lambda_q) and LW (mu; not read in the first stage):
// the fused kernel writes lambda_q and, unless the stage is the last one, the next mu to the
// partner buffers T1, T2 (inputs' halos are read by neighbouring CTAs), the ghost adjoints
// are scattered back into both, and the buffer pairs swap roles.
template <typename T>
static int enqueue_rhs_adjoint(solar_ctx* c, AdjStageArgs<T> a, bool last) {
  AdjBuffers& b = c->adj;
  const Geom& g = c->g;
  a.mu = (const T*)(a.first ? b.L : b.LW);
  a.lout = (T*)b.T1;
  a.muout = last ? nullptr : (T*)b.T2;
  if ((long long)g.nf * g.vs >= (1LL << 31))     // the kernel indexes one face's fields in 32 bits
    return fail(SOLAR_ERR_ARG, "grid too large for the adjoint (%lld values per face)", (long long)g.nf * g.vs);
  int rc = (g.n % 32 == 0) ? launch_adj_stage<T, 32, 8>(c, a) : launch_adj_stage<T, 16, 16>(c, a);
  if (rc) return rc;
  const AdjEdgeArgs<T> ae = {a.lout, a.muout, a.beta_next, (const T*)b.wt, b.wt_span, b.tspan, g, 0};
  CK(launch_pdl(adj_edge_kernel<T>, dim3(blocks_for(g.n, 128), 72, g.nr), dim3(128), 2 * g.n * sizeof(T), c->stream, ae));
  std::swap(b.L, b.T1);
  std::swap(b.LW, b.T2);
  return SOLAR_OK;
}

template <typename T, int TX, int TY, int R>
static int launch_adj_filter(solar_ctx* c) {
  using L = FilterLayout<T, TX, TY>;
  AdjBuffers& b = c->adj;
  const Geom& g = c->g;
  FilterArgs<T> a = {};
  if (!make_interior_map(c, b.L, TX + 8, TY + 6, &a.mP)) return fail(SOLAR_ERR_CUDA, "cuTensorMapEncodeTiled failed");
  a.qout = (T*)b.T1;
  a.runs = nullptr;
  a.wc = wait_ctl(c, kInjAdjFilter);
  a.g = g;
  constexpr int threads = (TX / Vec16<T>::V) * (TY / R);
  static bool attr_set = false;
  static int resident = 1;
  if (!attr_set) {
    CK(cudaFuncSetAttribute(adj_filter_kernel<T, TX, TY, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::TOTAL));
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, adj_filter_kernel<T, TX, TY, R>, threads, L::TOTAL));
    resident = std::max(resident, 1);
    attr_set = true;
  }
  const long long units = (long long)(g.n / TX) * (g.n / TY) * g.nf * 6;
  const long long grid = split_units(units, g.nr, c->nsm, resident, &a.whole, &a.chunks);
  CK(launch_pdl(adj_filter_kernel<T, TX, TY, R>, dim3((unsigned)grid), dim3(TX / Vec16<T>::V, TY / R), L::TOTAL, c->stream, a));
  return SOLAR_OK;
}

// FILTER_EXP^T on buffer L (which takes the scratch buffer's place and the other way round).
// The interior first: its kernel is the longer one and releases the next before its last planes (a
// reverse step at 6 x 32^2 x 24 in float 102.7 us the other way round, 96.4 this way).
template <typename T>
static int enqueue_filter_adjoint(solar_ctx* c) {
  const Geom& g = c->g;
  AdjBuffers& b = c->adj;
  AdjGhostArgs<T> a = {(const T*)b.L, (T*)b.T1, g, 16};             // 16 planes per thread
  const int warps = std::max((g.n + 31) / 32, (g.n + 25) / 26);     // a column warp writes 26 rows
  constexpr int R = sizeof(T) == 4 ? 1 : 2;                         // as launch_filter
  int rc = g.n % 32 == 0 ? launch_adj_filter<T, 32, 16, R>(c) : launch_adj_filter<T, 16, 16, R>(c);
  if (rc) return rc;
  CK(launch_pdl(adj_ghost_kernel<T>, dim3((unsigned)(warps + 3) / 4, (unsigned)((g.nr + a.kp - 1) / a.kp), 24 * g.nf), dim3(128),
                0, c->stream, a));
  std::swap(b.L, b.T1);
  const AdjEdgeArgs<T> ae = {(T*)b.L, nullptr, T(0), (const T*)b.wt, b.wt_span, b.tspan, g, 1};
  CK(launch_pdl(adj_edge_kernel<T>, dim3(blocks_for(g.n, 128), 72, g.nr), dim3(128), g.nf * g.n * sizeof(T), c->stream, ae));
  return SOLAR_OK;
}

// One reverse time step on buffer L: lambda_n -> lambda_{n-1}.  `dstep` holds the
// divergence of the five stage inputs of the forward step (gradient only).
template <typename T>
static int enqueue_step_adjoint(solar_ctx* c, const T* dstep, double* grad) {
  int rc;
  if ((rc = enqueue_filter_adjoint<T>(c))) return rc;
  const long long V6 = 6 * vol_compact(c);
  for (int s = 4; s >= 0; --s) {
    AdjStageArgs<T> a = adj_args<T>(c, c->desc.dt);
    a.first = s == 4;
    a.beta = s == 4 ? (T)kBeta[4] : T(1);
    a.alpha = (T)kAlpha[s];
    a.beta_next = s > 0 ? (T)kBeta[s - 1] : T(0);
    a.keep = 1;
    if (grad && dstep) { a.grad = grad; a.div = dstep + s * V6; }
    if ((rc = enqueue_rhs_adjoint<T>(c, a, s == 0))) return rc;
  }
  return SOLAR_OK;
}

// One forward step (same kernels as the step graph) that also stores the divergence of
// each stage input into dstep[stage][face][k][j][i].
template <typename T>
static int enqueue_step_div(solar_ctx* c, T* dstep) {
  void* bufs[2] = {c->A, c->B};
  const long long V6 = 6 * vol_compact(c);
  int cur = 0, rc;
  if ((rc = force_begin(c))) return rc;
  for (int s = 0; s < 5; ++s) {
    if ((rc = launch_edge<T>(c, bufs[cur], 0, nullptr))) return rc;
    if ((rc = launch_stage<T>(c, bufs[cur], bufs[cur ^ 1], s == 0 ? 4 : 5, s, nullptr, dstep + s * V6))) return rc;
    cur ^= 1;
  }
  if ((rc = launch_edge<T>(c, bufs[cur], 1, nullptr))) return rc;
  if ((rc = launch_filter<T>(c, bufs[cur], bufs[cur ^ 1], nullptr, true))) return rc;
  CK(cudaGetLastError());
  return SOLAR_OK;
}

template <typename T>
static void enqueue_sample(solar_ctx* c, double* out) {
  const AdjBuffers& b = c->adj;
  sample_kernel<T><<<blocks_for(b.nrec, 128), 128, 0, c->stream>>>((const T*)c->A, b.rec_off, b.rec_w, b.nrec, out);
}

// The checkpointed sweep.  Outer checkpoints every K steps are kept for the whole run.  With
// K2 < K each outer segment is first run forward again keeping inner checkpoints every K2
// steps, and each inner segment is then recomputed storing its stage-input divergences and
// reversed; memory is one state per outer and per inner checkpoint plus 5 * K2 field volumes,
// for one more forward run than the single-level sweep (K2 = K).
template <typename T>
static int misfit_gradient_t(solar_ctx* c, int N, int K, int K2, const double* data, double* misfit, double* grad_c,
                             double* lambda0, double* times) {
  AdjBuffers& b = c->adj;
  const long long V6 = 6 * vol_compact(c);
  const size_t S = (size_t)state_bytes(c);
  const int ncp = (N + K - 1) / K;
  K2 = std::max(1, std::min(K2, K));
  const int nsub_max = (std::min(K, N) + K2 - 1) / K2;
  int rc;
  if ((rc = adj_reserve(&b.ckpt, &b.ckpt_bytes, S * (size_t)ncp))) return rc;
  if (nsub_max > 1 && (rc = adj_reserve(&b.ckpt2, &b.ckpt2_bytes, S * (size_t)nsub_max))) return rc;
  if ((rc = adj_reserve(&b.div, &b.div_bytes, (size_t)std::min(K2, N) * 5 * V6 * sizeof(T)))) return rc;
  if ((rc = adj_reserve((void**)&b.traces, &b.traces_bytes, (size_t)std::max(N, 1) * b.nrec * 2 * sizeof(double)))) return rc;
  // with a source term the clock (time, step, interpolation state) is checkpointed too
  const size_t CL = sizeof(ForceClock);
  if (c->forcing && (rc = adj_reserve(&b.clk, &b.clk_bytes, CL * (size_t)(ncp + nsub_max)))) return rc;
  char* clk = (char*)b.clk;
  char* clk2 = clk + CL * (size_t)ncp;
  char* ckpt2 = (char*)b.ckpt2;
  double* traces = b.traces;
  double* res = b.traces + (size_t)N * b.nrec;
  char* ckpt = (char*)b.ckpt;
  T* D = (T*)b.div;
  if ((rc = capture_step_graph(c))) return rc;
  CK(cudaEventRecord(c->ev[2], c->stream));
  // forward sweep: checkpoints every K steps, receiver traces after every step
  for (int n = 0; n < N; ++n) {
    if (n % K == 0) {
      CK(cudaMemcpyAsync(ckpt + (size_t)(n / K) * S, c->A, S, cudaMemcpyDeviceToDevice, c->stream));
      if (c->forcing) CK(cudaMemcpyAsync(clk + (size_t)(n / K) * CL, c->force_clock, CL, cudaMemcpyDeviceToDevice, c->stream));
    }
    CK(cudaGraphLaunch(c->step_graph, c->stream));
    enqueue_sample<T>(c, traces + (size_t)n * b.nrec);
  }
  CK(cudaEventRecord(c->ev[3], c->stream));
  std::vector<double> h((size_t)N * b.nrec);
  CK(cudaMemcpyAsync(h.data(), traces, h.size() * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
  CK(cudaStreamSynchronize(c->stream));
  if ((rc = check_device_error(c))) return rc;
  double J = 0.0;
  for (size_t q = 0; q < h.size(); ++q) {
    h[q] -= data[q];
    J += 0.5 * h[q] * h[q];
  }
  if (misfit) *misfit = J;
  CK(cudaMemcpyAsync(res, h.data(), h.size() * sizeof(double), cudaMemcpyHostToDevice, c->stream));
  // reverse sweep, one checkpoint segment at a time
  CK(cudaMemsetAsync(c->adj.L, 0, S, c->stream));
  CK(cudaMemsetAsync(b.grad, 0, (size_t)V6 * sizeof(double), c->stream));
  float t_rec = 0.f, t_adj = 0.f;
  for (int seg = ncp - 1; seg >= 0; --seg) {
    const int n0 = seg * K, n1 = std::min(N, n0 + K);
    const int nsub = (n1 - n0 + K2 - 1) / K2;
    CK(cudaEventRecord(c->ev[4], c->stream));
    CK(cudaMemcpyAsync(c->A, ckpt + (size_t)seg * S, S, cudaMemcpyDeviceToDevice, c->stream));
    if (c->forcing) CK(cudaMemcpyAsync(c->force_clock, clk + (size_t)seg * CL, CL, cudaMemcpyDeviceToDevice, c->stream));
    if (nsub > 1)                  // inner checkpoints of this segment
      for (int n = n0; n < n1; ++n) {
        if ((n - n0) % K2 == 0) {
          const size_t q = (size_t)((n - n0) / K2);
          CK(cudaMemcpyAsync(ckpt2 + q * S, c->A, S, cudaMemcpyDeviceToDevice, c->stream));
          if (c->forcing) CK(cudaMemcpyAsync(clk2 + q * CL, c->force_clock, CL, cudaMemcpyDeviceToDevice, c->stream));
        }
        CK(cudaGraphLaunch(c->step_graph, c->stream));
      }
    CK(cudaEventRecord(c->ev[7], c->stream));
    CK(cudaEventSynchronize(c->ev[7]));
    float r0 = 0.f;
    CK(cudaEventElapsedTime(&r0, c->ev[4], c->ev[7]));
    t_rec += r0;
    for (int sub = nsub - 1; sub >= 0; --sub) {
      const int m0 = n0 + sub * K2, m1 = std::min(n1, m0 + K2);
      CK(cudaEventRecord(c->ev[4], c->stream));
      if (nsub > 1) {
        CK(cudaMemcpyAsync(c->A, ckpt2 + (size_t)sub * S, S, cudaMemcpyDeviceToDevice, c->stream));
        if (c->forcing) CK(cudaMemcpyAsync(c->force_clock, clk2 + (size_t)sub * CL, CL, cudaMemcpyDeviceToDevice, c->stream));
      }
      for (int n = m0; n < m1; ++n)
        if ((rc = enqueue_step_div<T>(c, D + (size_t)(n - m0) * 5 * V6))) return rc;
      CK(cudaEventRecord(c->ev[5], c->stream));
      for (int n = m1; n > m0; --n) {
        // lambda += S^T (S q_n - d_n), then lambda <- STEP^T lambda (with the gradient)
        inject_kernel<T><<<blocks_for(b.nrec, 128), 128, 0, c->stream>>>((T*)c->adj.L, b.rec_off, b.rec_w, b.nrec,
                                                                          res + (size_t)(n - 1) * b.nrec);
        if ((rc = enqueue_step_adjoint<T>(c, D + (size_t)(n - 1 - m0) * 5 * V6, b.grad))) return rc;
      }
      CK(cudaEventRecord(c->ev[6], c->stream));
      CK(cudaEventSynchronize(c->ev[6]));
      float a = 0.f, r = 0.f;
      CK(cudaEventElapsedTime(&r, c->ev[4], c->ev[5]));
      CK(cudaEventElapsedTime(&a, c->ev[5], c->ev[6]));
      t_rec += r;
      t_adj += a;
    }
  }
  grad_scale_kernel<T><<<blocks_for(V6, 256), 256, 0, c->stream>>>(b.grad, (const T*)c->dt.c2, (const T*)c->dt.radT, c->g.nr,
                                                                  (long long)c->g.n * c->g.n);
  CK(cudaGetLastError());
  // leave the state (and the clock) at the initial condition
  CK(cudaMemcpyAsync(c->A, ckpt, S, cudaMemcpyDeviceToDevice, c->stream));
  if (c->forcing) CK(cudaMemcpyAsync(c->force_clock, clk, CL, cudaMemcpyDeviceToDevice, c->stream));
  CK(cudaStreamSynchronize(c->stream));
  if ((rc = check_device_error(c))) return rc;
  if (times) {
    float f = 0.f;
    CK(cudaEventElapsedTime(&f, c->ev[2], c->ev[3]));
    times[0] = f;
    times[1] = t_rec;
    times[2] = t_adj;
  }
  if (grad_c) {
    const size_t bytes = (size_t)V6 * sizeof(double);
    if (bytes >= 8u << 20 && pageable_volumes(grad_c, bytes) && stage_download(c, grad_c, bytes)) {
      Staged st(c);
      if ((rc = st.out(grad_c, b.grad, bytes)) || (rc = st.finish())) return rc;
    } else {
      CK(cudaMemcpyAsync(grad_c, b.grad, bytes, cudaMemcpyDeviceToHost, c->stream));
    }
    CK(cudaStreamSynchronize(c->stream));
  }
  if (lambda0) return download_fields(c, c->adj.L, 0, lambda0, 5, kAllFields, 5);
  return SOLAR_OK;
}

}  // namespace solar

extern "C" {

int solar_gpu_set_receivers(solar_ctx* c, int nrec, const double* loc) {
  int rc = check_ctx(c);
  if (rc) return rc;
  if (nrec < 1 || !loc) return fail(SOLAR_ERR_ARG, "need nrec >= 1 and receiver locations");
  if ((rc = adj_alloc(c))) return rc;
  const Geom& g = c->g;
  std::vector<long long> off((size_t)nrec * 8);
  std::vector<double> w((size_t)nrec * 8);
  for (int r = 0; r < nrec; ++r) {
    const double f = loc[r * 4 + 0], x = loc[r * 4 + 1], y = loc[r * 4 + 2], z = loc[r * 4 + 3];
    const int face = (int)f;
    if (face != f || face < 0 || face > 5 || !(x >= 0 && x <= g.n - 1) || !(y >= 0 && y <= g.n - 1) ||
        !(z >= 0 && z <= g.nr - 1))
      return fail(SOLAR_ERR_ARG, "receiver %d outside the grid (face %g, i %g, j %g, k %g)", r, f, x, y, z);
    const int i0 = std::min((int)x, g.n - 2), j0 = std::min((int)y, g.n - 2), k0 = std::min((int)z, g.nr - 2);
    const double wx = x - i0, wy = y - j0, wz = z - k0;
    for (int cc = 0; cc < 8; ++cc) {
      const int di = cc & 1, dj = (cc >> 1) & 1, dk = cc >> 2;
      off[(size_t)r * 8 + cc] = g.vol(0, face, g.slot[kP]) + g.at(k0 + dk, j0 + dj, i0 + di);
      w[(size_t)r * 8 + cc] = (di ? wx : 1 - wx) * (dj ? wy : 1 - wy) * (dk ? wz : 1 - wz);
    }
  }
  AdjBuffers& b = c->adj;
  if (b.rec_off) cudaFree(b.rec_off);
  if (b.rec_w) cudaFree(b.rec_w);
  b.rec_off = nullptr;
  b.rec_w = nullptr;
  b.nrec = 0;
  CK(cudaMalloc((void**)&b.rec_off, off.size() * sizeof(long long)));
  CK(cudaMalloc((void**)&b.rec_w, w.size() * sizeof(double)));
  CK(cudaMemcpy(b.rec_off, off.data(), off.size() * sizeof(long long), cudaMemcpyHostToDevice));
  CK(cudaMemcpy(b.rec_w, w.data(), w.size() * sizeof(double), cudaMemcpyHostToDevice));
  b.nrec = nrec;
  return SOLAR_OK;
}

int solar_gpu_record(solar_ctx* c, int nsteps, double* traces) {
  int rc = check_ctx(c);
  if (rc) return rc;
  if (nsteps < 0 || !traces) return fail(SOLAR_ERR_ARG, "bad arguments");
  if (!c->adj.nrec) return fail(SOLAR_ERR_STATE, "no receivers set");
  AdjBuffers& b = c->adj;
  if ((rc = adj_reserve((void**)&b.traces, &b.traces_bytes, (size_t)std::max(nsteps, 1) * b.nrec * 2 * sizeof(double))))
    return rc;
  if ((rc = capture_step_graph(c))) return rc;
  for (int n = 0; n < nsteps; ++n) {
    CK(cudaGraphLaunch(c->step_graph, c->stream));
    if (c->fp32) enqueue_sample<float>(c, b.traces + (size_t)n * b.nrec);
    else enqueue_sample<double>(c, b.traces + (size_t)n * b.nrec);
  }
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(traces, b.traces, (size_t)nsteps * b.nrec * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
  CK(cudaStreamSynchronize(c->stream));
  return check_device_error(c);
}

int solar_gpu_misfit_gradient(solar_ctx* c, int nsteps, int checkpoint_every, const double* data,
                              double* misfit, double* grad_c, double* lambda0, double* times_ms) {
  return solar_gpu_misfit_gradient_nested(c, nsteps, checkpoint_every, checkpoint_every, data, misfit, grad_c,
                                          lambda0, times_ms);
}

int solar_gpu_misfit_gradient_nested(solar_ctx* c, int nsteps, int checkpoint_every, int inner_every,
                                     const double* data, double* misfit, double* grad_c, double* lambda0,
                                     double* times_ms) {
  int rc = check_ctx(c);
  if (rc) return rc;
  if (inner_every < 1) return fail(SOLAR_ERR_ARG, "need inner_every >= 1");
  if (nsteps < 1 || checkpoint_every < 1 || !data) return fail(SOLAR_ERR_ARG, "need nsteps >= 1, checkpoint_every >= 1 and data");
  if (!c->adj.nrec) return fail(SOLAR_ERR_STATE, "no receivers set");
  if ((rc = adj_alloc(c))) return rc;
  return c->fp32 ? misfit_gradient_t<float>(c, nsteps, checkpoint_every, inner_every, data, misfit, grad_c, lambda0, times_ms)
                 : misfit_gradient_t<double>(c, nsteps, checkpoint_every, inner_every, data, misfit, grad_c, lambda0, times_ms);
}

int solar_gpu_rhs_adjoint(solar_ctx* c, const double* mu, double* out) {
  int rc = check_ctx(c);
  if (rc) return rc;
  if (!mu || !out) return fail(SOLAR_ERR_ARG, "null array");
  if ((rc = adj_alloc(c))) return rc;
  if ((rc = upload_fields(c, c->adj.L, 0, mu, 5, kAllFields, 5))) return rc;
  rc = c->fp32 ? enqueue_rhs_adjoint<float>(c, adj_args<float>(c, 1.0), true)
               : enqueue_rhs_adjoint<double>(c, adj_args<double>(c, 1.0), true);
  if (rc) return rc;
  if ((rc = download_fields(c, c->adj.L, 0, out, 5, kAllFields, 5))) return rc;
  return check_device_error(c);
}

int solar_gpu_filter_adjoint(solar_ctx* c, const double* lam, double* out) {
  int rc = check_ctx(c);
  if (rc) return rc;
  if (!lam || !out) return fail(SOLAR_ERR_ARG, "null array");
  if ((rc = adj_alloc(c))) return rc;
  if ((rc = upload_fields(c, c->adj.L, 0, lam, 5, kAllFields, 5))) return rc;
  rc = c->fp32 ? enqueue_filter_adjoint<float>(c) : enqueue_filter_adjoint<double>(c);
  if (rc) return rc;
  if ((rc = download_fields(c, c->adj.L, 0, out, 5, kAllFields, 5))) return rc;
  return check_device_error(c);
}

int solar_gpu_rk4_adjoint(solar_ctx* c, int nsteps, const double* lam_in, double* lam_out) {
  int rc = check_ctx(c);
  if (rc) return rc;
  if (nsteps < 0 || !lam_in || !lam_out) return fail(SOLAR_ERR_ARG, "bad arguments");
  if ((rc = adj_alloc(c))) return rc;
  CK(cudaMemsetAsync(c->adj.L, 0, (size_t)state_bytes(c), c->stream));
  if ((rc = upload_fields(c, c->adj.L, 0, lam_in, 5, kAllFields, 5))) return rc;
  for (int n = 0; n < nsteps; ++n) {
    rc = c->fp32 ? enqueue_step_adjoint<float>(c, nullptr, nullptr) : enqueue_step_adjoint<double>(c, nullptr, nullptr);
    if (rc) return rc;
  }
  if ((rc = download_fields(c, c->adj.L, 0, lam_out, 5, kAllFields, 5))) return rc;
  return check_device_error(c);
}

}  // extern "C"
