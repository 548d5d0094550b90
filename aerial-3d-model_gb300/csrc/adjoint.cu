// Adjoint (vector-Jacobian products) of the reprojection + distortion
// residuals and the GPS-prior residuals, plus the per-observation Jacobians
// and the robust cost at a context's current state.
//
// Residuals (ba.rs:56-128):
//   e_k = u_k − π(K_g, R_c (X_p − C_c))           per observation in front
//   r_c = (C_c − prior_c) / σ_c  (per axis)       per camera with a prior
// Jacobians J = ∂π/∂θ are the reference's (ba.rs:79-98): left rotation
// perturbation R ← exp(ω) R, then the centre, the point and the intrinsics
// (f, cx, cy, k1, k2; the reference refines f, k1, k2).  The VJP returns
//   g_θ = Σ_k (∂e_k/∂θ)ᵀ λ_k + Σ_c (∂r_c/∂θ)ᵀ μ_c,   ∂e/∂θ = −J.
// The gradient of the robust cost is the VJP with λ_k = ρ'(|e_k|²)·2e_k and
// μ_c = 2 r_c.
#include <cstring>
#include <vector>

#include "context.cuh"
#include "lm_kernels.cuh"

namespace ba {
namespace {

constexpr unsigned T = 256;

// One observation's share of the VJP, in reverse mode: the cotangent goes
// back through the projection once instead of through Jacobian rows (63 FP64
// operations, 15 more where the cotangent is the cost's; the rows took 171).
struct ObsVjp {
  double rot[3];  // left perturbation of the rotation
  double pt[3];   // point; the centre's share is its negative
  double in[5];   // f, cx, cy, k1, k2
};

// cot: the caller's residual cotangents [2n], or null: those of the robust
// cost.  kGeo: rotation and point too.  Zero for an observation that is not
// in front of its camera.
template <bool kGeo>
__device__ __forceinline__ void obs_vjp(const Prob& P, const StateView& st, int64_t k, double sigma,
                                        const double* cot, ObsVjp& o) {
  const uint32_t cam = P.obs_cam[k];
  const double* R = st.rot + 9 * (size_t)cam;
  const double* K = st.intr + 5 * (size_t)P.cam_group[cam];
  double xc[3];
  bacam::to_cam(R, st.center + 3 * (size_t)cam, st.points + 3 * (size_t)P.obs_pt[k], xc);
  if (xc[2] <= 1e-6) {
#pragma unroll
    for (int i = 0; i < 3; ++i) o.rot[i] = o.pt[i] = 0.0;
#pragma unroll
    for (int i = 0; i < 5; ++i) o.in[i] = 0.0;
    return;
  }
  const double f = K[0], k1 = K[3], k2 = K[4];
  const double iz = __drcp_rn(xc[2]);
  const double px = mul_any(xc[0], iz), py = mul_any(xc[1], iz);
  const double r2 = sum2(px, px, py, py);
  const double d = fma(mul_any(k2, r2), r2, fma(k1, r2, 1.0));
  const double qx = mul_any(px, d), qy = mul_any(py, d);
  // e = u - pred: the prediction's cotangent is the residual's negative
  double l0, l1;
  if (cot) {
    l0 = -cot[2 * k], l1 = -cot[2 * k + 1];
  } else {  // d rho / d e = rho'(|e|^2) * 2 e, rho' = the IRLS weight
    const double ex = P.obs_uv[2 * k] - (f * qx + K[1]);
    const double ey = P.obs_uv[2 * k + 1] - (f * qy + K[2]);
    const double w = -2.0 * robust_weight(sum2(ex, ex, ey, ey), sigma, P.loss);
    l0 = mul_any(w, ex), l1 = mul_any(w, ey);
  }
  const double s = sum2(l0, px, l1, py);
  o.in[0] = sum2(l0, qx, l1, qy);
  o.in[1] = l0;
  o.in[2] = l1;
  o.in[3] = mul_any(mul_any(f, r2), s);
  o.in[4] = mul_any(o.in[3], r2);
  if constexpr (kGeo) {
    const double cs = mul_any(fma(4.0 * k2, r2, k1 + k1), s);
    const double fz = mul_any(f, iz);
    const double g0 = mul_any(sum2(d, l0, cs, px), fz), g1 = mul_any(sum2(d, l1, cs, py), fz);
    const double g2 = -sum2(g0, px, g1, py);
    o.rot[0] = fma(xc[1], g2, -mul_any(xc[2], g1));
    o.rot[1] = fma(xc[2], g0, -mul_any(xc[0], g2));
    o.rot[2] = fma(xc[0], g1, -mul_any(xc[1], g0));
#pragma unroll
    for (int j = 0; j < 3; ++j) o.pt[j] = fma(R[6 + j], g2, sum2(R[j], g0, R[3 + j], g1));
  }
}

__global__ void linearise_all_kernel(Prob P, StateView st, double sigma, double* out,
                                     const uint8_t* refine_model) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= P.no) return;
  double* o = out + (size_t)k * kLinW;
  const bool refine = refine_model[P.pt_model[P.obs_pt[k]]] != 0;
  if (!linearise<double>(P, st, k, sigma, refine, o))
    for (int i = 0; i < kLinW; ++i) o[i] = 0.0;
}

// Thread per point: its observations' contributions in order.
__global__ void vjp_point_kernel(Prob P, const uint32_t* pt_ptr, const double* gpt, double* out) {
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P.np) return;
  double a[3] = {0, 0, 0};
  for (uint32_t k = pt_ptr[p]; k < pt_ptr[p + 1]; ++k)
    for (int i = 0; i < 3; ++i) a[i] += gpt[3 * (size_t)k + i];
  for (int i = 0; i < 3; ++i) out[3 * p + i] = a[i];
}

// A quarter of a camera's observations per CTA, in camera order: their shares
// of the camera and its intrinsics summed, the points' stored (24 bytes an
// observation; with a pass of its own per observation, 112 and read again).
// Bound by the FP64 operations, whose plain products are made in integers (2.6 M
// observations: 0.48 -> 0.37 ms); quarters, because 500 cameras on 152 SMs would
// leave the last wave a third full.
constexpr int kVjpThreads = 128;
constexpr int kVjpParts = 4;
constexpr int kVjpN = 11;  // rotation 3, centre 3, intrinsics 5

__global__ void __launch_bounds__(kVjpThreads)
    vjp_camera_kernel(Prob P, StateView st, const uint32_t* cam_ptr, const uint32_t* cam_obs,
                      double sigma, const double* cot, double* gpt, double* part) {
  __shared__ double scratch[kVjpN * 32];
  const int64_t c = blockIdx.x / kVjpParts, q = blockIdx.x % kVjpParts;
  const uint32_t c0 = cam_ptr[c], n = cam_ptr[c + 1] - c0;
  const uint32_t b = c0 + (uint32_t)((uint64_t)n * q / kVjpParts);
  const uint32_t e = c0 + (uint32_t)((uint64_t)n * (q + 1) / kVjpParts);
  double a[kVjpN];
#pragma unroll
  for (int i = 0; i < kVjpN; ++i) a[i] = 0.0;
  for (uint32_t i = b + threadIdx.x; i < e; i += kVjpThreads) {
    const uint32_t k = cam_obs[i];
    ObsVjp o;
    obs_vjp<true>(P, st, k, sigma, cot, o);
    if (gpt)
#pragma unroll
      for (int t = 0; t < 3; ++t) gpt[3 * (size_t)k + t] = o.pt[t];
#pragma unroll
    for (int t = 0; t < 3; ++t) a[t] += o.rot[t], a[3 + t] -= o.pt[t];
#pragma unroll
    for (int t = 0; t < 5; ++t) a[6 + t] += o.in[t];
  }
  block_sum<kVjpN>(a, scratch);
  if (threadIdx.x == 0)
    for (int t = 0; t < kVjpN; ++t) part[(size_t)blockIdx.x * kVjpN + t] = a[t];
}

// Thread per camera: its quarters in order, plus the prior term.
__global__ void vjp_camera_sum_kernel(Prob P, StateView st, const double* part,
                                      const double* cot_prior, double* out_cam,
                                      double* out_cam_int) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= P.nc) return;
  double a[kVjpN];
#pragma unroll
  for (int t = 0; t < kVjpN; ++t) {
    a[t] = 0.0;
    for (int q = 0; q < kVjpParts; ++q) a[t] += part[(size_t)(kVjpParts * c + q) * kVjpN + t];
  }
  if (P.prior_mask && P.prior_mask[c]) {
    const double* q = P.prior + 6 * (size_t)c;
    for (int t = 0; t < 3; ++t) {
      const double r = (st.center[3 * c + t] - q[t]) / q[3 + t];
      const double mu = cot_prior ? cot_prior[3 * c + t] : 2.0 * r;
      a[3 + t] += mu / q[3 + t];
    }
  }
#pragma unroll
  for (int t = 0; t < 6; ++t) out_cam[6 * c + t] = a[t];
#pragma unroll
  for (int t = 0; t < 5; ++t) out_cam_int[5 * c + t] = a[6 + t];
}

// Intrinsics alone, models of one lens group each: a chunk of a model's
// observations per CTA, in observation order (no index by camera is built),
// then a model's chunks by a CTA.
__global__ void __launch_bounds__(kCostThreads)
    vjp_chunk_kernel(Prob P, StateView st, StructView S, double sigma, const double* cot,
                     double* part) {
  __shared__ double scratch[5 * 32];
  double a[5] = {0, 0, 0, 0, 0};
  for (uint32_t k = S.cost_chunk_begin[blockIdx.x] + threadIdx.x;
       k < S.cost_chunk_end[blockIdx.x]; k += kCostThreads) {
    ObsVjp o;
    obs_vjp<false>(P, st, k, sigma, cot, o);
#pragma unroll
    for (int t = 0; t < 5; ++t) a[t] += o.in[t];
  }
  block_sum<5>(a, scratch);
  if (threadIdx.x == 0)
    for (int t = 0; t < 5; ++t) part[5 * (size_t)blockIdx.x + t] = a[t];
}

__global__ void __launch_bounds__(kCostFinalThreads)
    vjp_chunk_sum_kernel(StructView S, const double* part, const uint32_t* group, double* out) {
  __shared__ double scratch[5 * 32];
  const int64_t m = blockIdx.x;
  double a[5] = {0, 0, 0, 0, 0};
  for (uint32_t c = S.model_chunk0[m] + threadIdx.x; c < S.model_chunk0[m + 1];
       c += kCostFinalThreads)
    for (int t = 0; t < 5; ++t) a[t] += part[5 * (size_t)c + t];
  block_sum<5>(a, scratch);
  if (threadIdx.x == 0 && group[m + 1] > group[m])
    for (int t = 0; t < 5; ++t) out[5 * (size_t)group[m] + t] = a[t];
}

__global__ void vjp_group_kernel(Prob P, const uint32_t* grp_ptr, const uint32_t* grp_cams,
                                 const double* cam_int, double* out) {
  const int64_t g = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (g >= P.ng) return;
  double a[5] = {0, 0, 0, 0, 0};
  for (uint32_t i = grp_ptr[g] + lane; i < grp_ptr[g + 1]; i += 32)
    for (int t = 0; t < 5; ++t) a[t] += cam_int[5 * (size_t)grp_cams[i] + t];
  for (int t = 0; t < 5; ++t) a[t] = warp_sum(a[t]);
  if (lane == 0)
    for (int t = 0; t < 5; ++t) out[5 * g + t] = a[t];
}

void require(const Context& c) {
  if (!c.uploaded) throw BadInput("no problem uploaded");
  check(cudaSetDevice(c.device), "cudaSetDevice");
}

// Cost chunks aligned to model boundaries (the solver's cost plan).
struct CostPlan {
  DevBuf<uint32_t> model, begin, end, m0;
  int64_t n = 0;
  StructView view() const {
    StructView v{};
    v.cost_chunk_model = model;
    v.cost_chunk_begin = begin;
    v.cost_chunk_end = end;
    v.model_chunk0 = m0;
    v.ncost = n;
    return v;
  }
};

void make_cost_plan(const Context& c, CostPlan& pl) {
  constexpr uint32_t CH = 4096;
  std::vector<uint32_t> cm, cb, ce, m0(c.nm + 1);
  for (int64_t m = 0; m < c.nm; ++m) {
    m0[m] = (uint32_t)cm.size();
    uint32_t x = c.h_obs0[m];
    const uint32_t e = c.h_obs0[m + 1];
    do {
      cm.push_back((uint32_t)m), cb.push_back(x), ce.push_back(std::min(e, x + CH));
      x += CH;
    } while (x < e);
  }
  m0[c.nm] = (uint32_t)cm.size();
  pl.n = (int64_t)cm.size();
  cudaStream_t s = c.stream;
  pl.model.alloc(pl.n, s), pl.begin.alloc(pl.n, s), pl.end.alloc(pl.n, s), pl.m0.alloc(c.nm + 1, s);
  check(cudaMemcpyAsync(pl.model, cm.data(), 4 * cm.size(), cudaMemcpyHostToDevice, s), "h2d");
  check(cudaMemcpyAsync(pl.begin, cb.data(), 4 * cb.size(), cudaMemcpyHostToDevice, s), "h2d");
  check(cudaMemcpyAsync(pl.end, ce.data(), 4 * ce.size(), cudaMemcpyHostToDevice, s), "h2d");
  check(cudaMemcpyAsync(pl.m0, m0.data(), 4 * m0.size(), cudaMemcpyHostToDevice, s), "h2d");
  check(cudaStreamSynchronize(s), "cost plan");
}

void context_cost(Context& c, const ba_options* opt, double* cost, double* rms, int64_t* nf) {
  require(c);
  const Opts o = resolve_options(opt);
  cudaStream_t s = c.stream;
  const Prob P = c.prob(o.loss);
  CostPlan pl;
  make_cost_plan(c, pl);
  const StructView SV = pl.view();
  DevBuf<double> part(std::max<int64_t>(pl.n, 1) * 3, s), sg(c.nm, s), dc(c.nm, s), dsq(c.nm, s);
  DevBuf<int64_t> dn(c.nm, s);
  std::vector<double> h_sg(c.nm, o.sigma);
  check(cudaMemcpyAsync(sg.p, h_sg.data(), 8 * c.nm, cudaMemcpyHostToDevice, s), "h2d");
  BA_LAUNCH(cost_chunk_kernel<<<(unsigned)std::max<int64_t>(pl.n, 1), kCostThreads, 0, s>>>(
      P, c.cur(), SV, part, nullptr, sg));
  BA_LAUNCH(cost_final_kernel<<<(unsigned)c.nm, kCostFinalThreads, 0, s>>>(P, c.cur(), SV, part,
                                                                      nullptr, dc, dsq, dn));
  std::vector<double> hc(c.nm), hsq(c.nm);
  std::vector<int64_t> hn(c.nm);
  check(cudaMemcpyAsync(hc.data(), dc.p, 8 * c.nm, cudaMemcpyDeviceToHost, s), "d2h");
  check(cudaMemcpyAsync(hsq.data(), dsq.p, 8 * c.nm, cudaMemcpyDeviceToHost, s), "d2h");
  check(cudaMemcpyAsync(hn.data(), dn.p, 8 * c.nm, cudaMemcpyDeviceToHost, s), "d2h");
  check(cudaStreamSynchronize(s), "cost");
  for (int64_t m = 0; m < c.nm; ++m) {
    if (cost) cost[m] = hc[m];
    if (rms) rms[m] = std::sqrt(hsq[m] / (double)std::max<int64_t>(hn[m], 1));
    if (nf) nf[m] = hn[m];
  }
}

void context_linearise(Context& c, const ba_options* opt, double* e, double* jc, double* jg,
                       double* jp, double* w, uint8_t* valid) {
  require(c);
  const Opts o = resolve_options(opt);
  cudaStream_t s = c.stream;
  const int64_t no = c.no;
  if (no == 0) return;
  DevBuf<double> out(no * kLinW, s);
  BA_LAUNCH(linearise_all_kernel<<<grid_for(no, T), T, 0, s>>>(c.prob(o.loss), c.cur(), o.sigma,
                                                              out, c.model_refine));
  std::vector<double> h(no * kLinW);
  check(cudaMemcpyAsync(h.data(), out.p, 8 * h.size(), cudaMemcpyDeviceToHost, s), "d2h");
  check(cudaStreamSynchronize(s), "linearise");
  for (int64_t k = 0; k < no; ++k) {
    const double* r = h.data() + k * kLinW;
    if (e) std::memcpy(e + 2 * k, r + 24, 16);
    if (jc) std::memcpy(jc + 12 * k, r, 96);
    if (jp) std::memcpy(jp + 6 * k, r + 12, 48);
    if (jg) std::memcpy(jg + 6 * k, r + 18, 48);
    if (w) w[k] = r[26];
    if (valid) valid[k] = r[27] != 0.0 ? 1 : 0;
  }
}

void context_vjp(Context& c, const ba_options* opt, const double* cot_obs,
                 const double* cot_prior, double* g_cam, double* g_pt, double* g_intr) {
  require(c);
  const Opts o = resolve_options(opt);
  cudaStream_t s = c.stream;
  const Prob P = c.prob(o.loss);
  const int64_t no = c.no, nc = c.nc, np = c.np, ng = c.ng;
  DevBuf<double> d_cot(cot_obs ? 2 * no : 0, s), d_cotp(cot_prior ? 3 * nc : 0, s);
  if (cot_obs && no)
    check(cudaMemcpyAsync(d_cot.p, cot_obs, 16 * no, cudaMemcpyHostToDevice, s), "h2d");
  if (cot_prior && nc)
    check(cudaMemcpyAsync(d_cotp.p, cot_prior, 24 * nc, cudaMemcpyHostToDevice, s), "h2d");
  const double* cot = cot_obs ? d_cot.p : nullptr;
  DevBuf<double> og(std::max<int64_t>(ng, 1) * 5, s);
  bool one_group = true;
  for (int64_t m = 0; m < c.nm; ++m) one_group = one_group && c.h_grp0[m + 1] - c.h_grp0[m] <= 1;
  if (!g_cam && !g_pt && one_group) {
    CostPlan pl;
    make_cost_plan(c, pl);
    DevBuf<double> part(5 * (size_t)pl.n, s);
    DevBuf<uint32_t> grp0(c.nm + 1, s);
    check(cudaMemcpyAsync(grp0.p, c.h_grp0.data(), 4 * (c.nm + 1), cudaMemcpyHostToDevice, s), "h2d");
    BA_LAUNCH(vjp_chunk_kernel<<<(unsigned)pl.n, kCostThreads, 0, s>>>(P, c.cur(), pl.view(),
                                                                      o.sigma, cot, part));
    BA_LAUNCH(vjp_chunk_sum_kernel<<<(unsigned)c.nm, kCostFinalThreads, 0, s>>>(pl.view(), part,
                                                                               grp0, og));
    if (g_intr && ng) check(cudaMemcpyAsync(g_intr, og.p, 40 * ng, cudaMemcpyDeviceToHost, s), "d2h");
    check(cudaStreamSynchronize(s), "vjp");
    return;
  }
  StructBufs SB;
  build_cam_index(P, SB, s);
  DevBuf<double> gp(std::max<int64_t>(g_pt ? 3 * no : 1, 1), s);
  DevBuf<double> oc(std::max<int64_t>(nc, 1) * 6, s), oci(std::max<int64_t>(nc, 1) * 5, s),
      part(std::max<int64_t>(nc, 1) * kVjpParts * kVjpN, s), op(std::max<int64_t>(np, 1) * 3, s);
  if (nc) {
    BA_LAUNCH(vjp_camera_kernel<<<(unsigned)(nc * kVjpParts), kVjpThreads, 0, s>>>(
        P, c.cur(), SB.cam_ptr, SB.cam_obs, o.sigma, cot, g_pt ? gp.p : nullptr, part));
    BA_LAUNCH(vjp_camera_sum_kernel<<<grid_for(nc, 128), 128, 0, s>>>(
        P, c.cur(), part, cot_prior ? d_cotp.p : nullptr, oc, oci));
  }
  if (np && g_pt) {
    SB.pt_ptr.alloc(np + 1, s);
    lower_bounds_u32(P.obs_pt, no, SB.pt_ptr, np, s);
    BA_LAUNCH(vjp_point_kernel<<<grid_for(np, T), T, 0, s>>>(P, SB.pt_ptr, gp, op));
  }
  if (ng)
    BA_LAUNCH(vjp_group_kernel<<<grid_for(ng * 32, 128), 128, 0, s>>>(P, SB.grp_ptr, SB.grp_cams,
                                                                     oci, og));
  if (g_cam && nc) check(cudaMemcpyAsync(g_cam, oc.p, 48 * nc, cudaMemcpyDeviceToHost, s), "d2h");
  if (g_pt && np) check(cudaMemcpyAsync(g_pt, op.p, 24 * np, cudaMemcpyDeviceToHost, s), "d2h");
  if (g_intr && ng) check(cudaMemcpyAsync(g_intr, og.p, 40 * ng, cudaMemcpyDeviceToHost, s), "d2h");
  check(cudaStreamSynchronize(s), "vjp");
}

}  // namespace
}  // namespace ba

using namespace ba;

extern "C" {

ba_status ba_context_cost(ba_context* c, const ba_options* opt, double* cost, double* rms,
                          int64_t* n_in_front) {
  if (!c) return set_error(BA_BAD_INPUT, "null context");
  return guarded([&] { context_cost(*c, opt, cost, rms, n_in_front); });
}

ba_status ba_context_linearise(ba_context* c, const ba_options* opt, double* e, double* jc,
                               double* jg, double* jp, double* w, uint8_t* valid) {
  if (!c) return set_error(BA_BAD_INPUT, "null context");
  return guarded([&] { context_linearise(*c, opt, e, jc, jg, jp, w, valid); });
}

ba_status ba_context_vjp(ba_context* c, const ba_options* opt, const double* cot_obs,
                         const double* cot_prior, double* g_cam, double* g_points,
                         double* g_intr) {
  if (!c) return set_error(BA_BAD_INPUT, "null context");
  return guarded([&] { context_vjp(*c, opt, cot_obs, cot_prior, g_cam, g_points, g_intr); });
}

ba_status ba_context_intrinsics_grad(ba_context* c, const ba_options* opt, double* grad) {
  if (!c) return set_error(BA_BAD_INPUT, "null context");
  if (!grad) return set_error(BA_BAD_INPUT, "null gradient array");
  return guarded([&] { context_vjp(*c, opt, nullptr, nullptr, nullptr, nullptr, grad); });
}

}  // extern "C"
