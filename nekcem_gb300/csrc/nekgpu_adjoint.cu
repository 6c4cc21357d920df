// Discrete adjoint of the FP64 fused stage (nekgpu_fp64.cu) with
// respect to the state and to the permittivity eps at every node.
//
// Forward stage i (src/cem_maxwell.F:484-508, src/cem_common.F:18-75):
//   r_i = M^-1(eps) (A(eps) u_{i-1} + s(t_i)),  k_i = a_i k_{i-1} + dt r_i,
//   u_i = u_{i-1} + b_i k_i,
// A = weighted curl (src/cem_maxwell.F:1428-1497) + upwind face flux with the
// partner face (src/cem_maxwell.F:922-1002) + lift; M^-1 = diag(hbm1, ebm1),
// ebm1 = 1/(eps bm1); the face impedance coefficients depend on eps at the
// node and at its partner (src/cem_maxwell.F:262-325).
//
// Reverse stage i carries (ub_i, w_i) with w_i = dt M^-1 (kb_i + b_i ub_i),
// kb_i the adjoint of k_i:
//   ub_{i-1} = ub_i + A^T w_i
//   w_{i-1}  = a_i w_i + b_{i-1} dt M^-1 ub_{i-1}      (kb_{i-1} = a_i kt_i)
//   deps    += -(bm1/dt) sum_E w_i,E (k_i - a_i k_{i-1})_E   (d ebm1/d eps)
//            + w_i^T (dA/deps) u_{i-1}                      (face impedances)
// A^T: the curl transposes to D^T contractions of w3 w; a face node's flux
// term L (u+ - u-) transposes to -L^T w at the node and +L^T w at its partner,
// and only the two tangential components of H and E enter (the normal one is
// projected out).  Every element gathers what lands on its own nodes, reading
// the partner elements' face nodes, so all writes are element-local: no
// atomics, and the adjoint state ping-pongs like the forward state.
//
// The kernel has the forward stage's form (nekgpu_fp64.cu): the weights w of
// an element in shared memory, one thread per face node, then two phases of
// line tasks (D^T w3 w in 64-bit integer arithmetic, nekgpu_fixed.cuh), both
// adding to ub in shared memory, then node by node the updates of w and deps
// in FP64.  The face terms (16 coefficients, the stage weights and the jumps)
// run in double-float FP32 arithmetic: float pairs, products with their FMA
// error terms, two-sum accumulation, ~2^-47 of the sum of the magnitudes, each
// result joined into one FP64 value.
//
// What bounds it: latencies at four blocks per SM, the FP64 pipe (41 slots per
// node) 42 % and issue (74 warp instructions per node, the face terms most of
// them) 39 % busy; 49 us per stage at 512 elements, N=7.  With double-float
// contractions per node and the face terms added per node by divergent warps
// (~100 FP64 slots per node, 512 threads and one block per SM) the reverse
// sweep of 100 steps of the 8^3-element N=7 box, the recomputation beside it,
// took 45 ms; it takes 32 ms.
#include <cuda_runtime.h>

#include "nekgpu_internal.h"
#include "nekgpu_lines.cuh"
#include "nekgpu_pair.cuh"

namespace nekgpu {

namespace {

// tangential axes in cyclic order: (e_a x x)_t1 = -x_t2, (e_a x x)_t2 = x_t1
__host__ __device__ constexpr int tan1(int a) { return a == 0 ? 1 : (a == 1 ? 2 : 0); }
__host__ __device__ constexpr int tan2(int a) { return a == 0 ? 2 : (a == 1 ? 0 : 1); }

// double-float values: (h, l) with h + l the value to ~2^-48
struct P2 {
  float h, l;
};
__device__ __forceinline__ P2 p2(double d) { return P2{d2f_hi(d), d2f_lo(d)}; }
__device__ __forceinline__ P2 p2(float2 v) { return P2{v.x, v.y}; }
__device__ __forceinline__ P2 pmul(P2 a, P2 b) {
  const float p = a.h * b.h;
  float e = fmaf(a.h, b.h, -p);
  e = fmaf(a.h, b.l, e);
  e = fmaf(a.l, b.h, e);
  return P2{p, e};
}
__device__ __forceinline__ P2 padd(P2 a, P2 b) {
  float s, t;
  two_sum(a.h, b.h, s, t);
  return P2{s, (a.l + b.l) + t};
}
__device__ __forceinline__ P2 pneg(P2 a) { return P2{-a.h, -a.l}; }
__device__ __forceinline__ double pdbl(P2 a) {
  float s, t;
  two_sum(a.h, a.l, s, t);
  return pair_to_double(s, t);
}

// WIDE: a thread per node, line and face node (dispatch_adjoint)
template <int NX, bool WIDE>
struct ACfg : ElemCfg<NX> {
  using E = ElemCfg<NX>;
  static constexpr int NT = WIDE ? round32(cmax(E::N3, E::NF)) : E::NT;
  static constexpr int FPT = (E::NF + NT - 1) / NT;
  // weights w; ub, completed in place; products of two GLL weights: 56 KB at
  // N=7, four blocks per SM
  static constexpr size_t off_R = 6 * (size_t)E::N3P * 8, off_w = 2 * off_R;
  static constexpr size_t smem = off_w + (size_t)E::N2 * 8;
};

// Phase PH of the transposed curl: every line adds its outputs, times the
// line's factor metric * w * w, to ub.
template <int NX, int PH, int NT>
__device__ __forceinline__ void adjoint_lines(const double* s_w, double* s_R, const double* s_ww,
                                              const double* eg, const AdjointDev& a) {
  using C = ElemCfg<NX>;
  constexpr int N2 = C::N2;
#pragma unroll 1
  for (int task = threadIdx.x; task < 6 * N2; task += NT) {
    const int type = task / N2, lam = task - type * N2;
    const LineType& lt = kLine[PH][type];
    const int dir = lt.dir, la = lam % NX, lb = lam / NX;
    const int base = dir == 0 ? C::RS * la + C::SZ * lb : (dir == 1 ? la + C::SZ * lb : la + C::RS * lb);
    const int step = dir == 0 ? 1 : (dir == 1 ? C::RS : C::SZ);
    const double rho = flip(eg[dir] * s_ww[lam], lt.neg != 0);
    double* R = s_R + lt.res * C::N3P + base;
    line_outputs<NX, false>(s_w + lt.comp * C::N3P + base, step, 0, NX, a.fd, a.Dw, nullptr,
                            [&](int i, double x) { R[step * i] = fma(rho, x, R[step * i]); });
  }
}

template <int NX, bool WIDE>
constexpr int adjoint_min_blocks() {
  return WIDE ? 1 : (NX == 9 ? 2 : 4);
}

template <int NX, bool WIDE>
__global__ void __launch_bounds__(ACfg<NX, WIDE>::NT, adjoint_min_blocks<NX, WIDE>())
    k_adjoint_stage(const __grid_constant__ AdjointDev a) {
  using C = ACfg<NX, WIDE>;
  constexpr int N2 = C::N2, N3 = C::N3, NT = C::NT, NF = C::NF, N3P = C::N3P;
  extern __shared__ __align__(16) unsigned char smem[];
  double* s_w = reinterpret_cast<double*>(smem);
  double* s_R = reinterpret_cast<double*>(smem + C::off_R);
  double* s_ww = reinterpret_cast<double*>(smem + C::off_w);
  const int tid = threadIdx.x;
  const long P = a.npts, PF = (long)a.nelt * NF;
  for (int t = tid; t < N2; t += NT) s_ww[t] = a.w[t % NX] * a.w[t / NX];
  const float2* kslot = reinterpret_cast<const float2*>(a.slot);
  // a programmatic dependent of the launch before: nothing it wrote is read,
  // and nothing it reads is written, before it has completed.  The next launch
  // may start from the last element's updates on; its blocks wait there beside
  // the recomputation's (us per reverse stage with the recomputation, without /
  // with: N=4 4 elements 16.5 / 14.4, N=7 64 elements 26.5 / 24.1, 512 elements
  // 67.7 / 67.0).
  asm volatile("griddepcontrol.wait;\n" ::: "memory");

  for (int e = blockIdx.x; e < a.nelt; e += gridDim.x) {
    const long ge = (long)e * N3;
    for (int v = tid; v < N3; v += NT) {
      const int pv = pnode<NX>(v);
#pragma unroll
      for (int c = 0; c < 6; ++c) {
        cp_async8(s_w + c * N3P + pv, a.w_in + c * P + ge + v);
        cp_async8(s_R + c * N3P + pv, a.ub_in + c * P + ge + v);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    // ---- face slots: transposed flux and impedance derivatives --------------
    // (the face node's share of deps; its terms of the component that waits)
    double fe[C::FPT], later[C::FPT][2];
#pragma unroll
    for (int q = 0; q < C::FPT; ++q) {
      const int t = tid + q * NT;
      fe[q] = 0.0;
      if (t >= NF) continue;
      const int f = t / N2, ab = t - f * N2, fa = ab % NX, fb = ab / NX;
      const int ax = slot_axis(f), t1 = tan1(ax), t2 = tan2(ax);
      const int vl = face_vol<NX>(f, fa, fb), pv = pnode<NX>(vl);
      const long gn = ge + vl, j = (long)e * NF + t;
      const int pe = a.nbr[6 * e + f];
      auto k = [&](int m) { return p2(kslot[m * PF + j]); };
      // own stage weights, and the jump u+ - u- of u_{i-1} (PEC: u-, the -2 of
      // the mirror is in the coefficients), tangential components
      const P2 nH1 = p2(s_w[t1 * N3P + pv]), nH2 = p2(s_w[t2 * N3P + pv]);
      const P2 nE1 = p2(s_w[(3 + t1) * N3P + pv]), nE2 = p2(s_w[(3 + t2) * N3P + pv]);
      P2 pH1{0.0f, 0.0f}, pH2{0.0f, 0.0f}, pE1{0.0f, 0.0f}, pE2{0.0f, 0.0f};
      P2 dH1 = p2(a.u_prev[t1 * P + gn]), dH2 = p2(a.u_prev[t2 * P + gn]);
      P2 dE1 = p2(a.u_prev[(3 + t1) * P + gn]), dE2 = p2(a.u_prev[(3 + t2) * P + gn]);
      if (pe >= 0) {
        const long gp = (long)pe * N3 + face_vol<NX>(slot_opp(f), fa, fb);
        pH1 = p2(a.w_in[t1 * P + gp]);
        pH2 = p2(a.w_in[t2 * P + gp]);
        pE1 = p2(a.w_in[(3 + t1) * P + gp]);
        pE2 = p2(a.w_in[(3 + t2) * P + gp]);
        dH1 = padd(p2(a.u_prev[t1 * P + gp]), pneg(dH1));
        dH2 = padd(p2(a.u_prev[t2 * P + gp]), pneg(dH2));
        dE1 = padd(p2(a.u_prev[(3 + t1) * P + gp]), pneg(dE1));
        dE2 = padd(p2(a.u_prev[(3 + t2) * P + gp]), pneg(dE2));
      }
      // Each component takes terms from the faces of its two tangential axes:
      // from those of the axis after it (it is their t2) now, from the other
      // axis' (their t1) after a barrier, so no two threads meet at a node.
      double* R = s_R + t2 * N3P + pv;
      // k: 0 kH 1 kHx 2 kE 3 kEx | 4 pH 5 pHx 6 pE 7 pEx | 8..11 gA..gD | 12..15 hA..hD
      {
        const P2 kH = k(0), kHx = k(1), qH = k(4), qHx = k(5);
        later[q][0] = pdbl(padd(padd(pmul(kH, nH1), pneg(pmul(kHx, nE2))),
                                padd(pmul(qH, pH1), pneg(pmul(qHx, pE2)))));
        R[0] += pdbl(padd(padd(pmul(kH, nH2), pmul(kHx, nE1)),
                          padd(pmul(qH, pH2), pmul(qHx, pE1))));
      }
      {
        const P2 kE = k(2), kEx = k(3), qE = k(6), qEx = k(7);
        later[q][1] = pdbl(padd(padd(pneg(pmul(kEx, nH2)), pmul(kE, nE1)),
                                padd(pneg(pmul(qEx, pH2)), pmul(qE, pE1))));
        R[3 * N3P] += pdbl(padd(padd(pmul(kEx, nH1), pmul(kE, nE2)),
                                padd(pmul(qEx, pH1), pmul(qE, pE2))));
      }
      // fe = A.PdH + B.(e_a x dE) + C.(e_a x dH) + D.PdE with A = gA wH(n) + hA wH(p) ...
      P2 F;
      {
        const P2 g = k(8), h = k(12);
        F = pmul(padd(pmul(g, nH1), pmul(h, pH1)), dH1);
        F = padd(F, pmul(padd(pmul(g, nH2), pmul(h, pH2)), dH2));
      }
      {
        const P2 g = k(9), h = k(13);
        F = padd(F, pneg(pmul(padd(pmul(g, nH1), pmul(h, pH1)), dE2)));
        F = padd(F, pmul(padd(pmul(g, nH2), pmul(h, pH2)), dE1));
      }
      {
        const P2 g = k(10), h = k(14);
        F = padd(F, pneg(pmul(padd(pmul(g, nE1), pmul(h, pE1)), dH2)));
        F = padd(F, pmul(padd(pmul(g, nE2), pmul(h, pE2)), dH1));
      }
      {
        const P2 g = k(11), h = k(15);
        F = padd(F, pmul(padd(pmul(g, nE1), pmul(h, pE1)), dE1));
        F = padd(F, pmul(padd(pmul(g, nE2), pmul(h, pE2)), dE2));
      }
      fe[q] = pdbl(F);
    }
    // after the barrier the other component, and the faces' deps one axis after
    // the other beside the phases (an axis' two faces share no node)
    auto each_face = [&](auto fn) {
#pragma unroll
      for (int q = 0; q < C::FPT; ++q) {
        const int t = tid + q * NT, f = t / N2;
        if (t < NF) fn(q, slot_axis(f), face_vol<NX>(f, (t - f * N2) % NX, (t - f * N2) / NX));
      }
    };
    auto face_deps = [&](int axis) {
      each_face([&](int q, int ax, int vl) {
        if (ax == axis) a.deps[ge + vl] += fe[q];
      });
    };
    const double* eg = a.egeom + 9 * (long)e;
    face_deps(0);
    __syncthreads();
    each_face([&](int q, int ax, int vl) {
      double* R = s_R + tan1(ax) * N3P + pnode<NX>(vl);
      R[0] += later[q][0];
      R[3 * N3P] += later[q][1];
    });
    face_deps(1);
    __syncthreads();
    face_deps(2);
    adjoint_lines<NX, 0, NT>(s_w, s_R, s_ww, eg, a);
    __syncthreads();
    adjoint_lines<NX, 1, NT>(s_w, s_R, s_ww, eg, a);
    __syncthreads();
    if (e + (int)gridDim.x >= a.nelt) asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    // ---- updates of ub, w and deps, node by node --------------------------------
#pragma unroll 1
    for (int v = tid; v < N3; v += NT) {
      const int pv = pnode<NX>(v);
      const long g = ge + v;
      double kc[3], kp[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        kc[c] = a.k_cur[(3 + c) * P + g];
        kp[c] = a.a == 0.0 ? 0.0 : a.k_prev[(3 + c) * P + g];
      }
      const double cH = a.bdt_next * a.hbm1[g], cE = a.bdt_next * a.ebm1[g];
      const double bm = -a.bm1[g] * a.inv_dt, d0 = a.deps[g];
      double mass = 0.0;
#pragma unroll
      for (int c = 0; c < 6; ++c) {
        const double wn = s_w[c * N3P + pv], out = s_R[c * N3P + pv];
        if (c >= 3) mass = fma(wn, a.a == 0.0 ? kc[c - 3] : fma(-a.a, kp[c - 3], kc[c - 3]), mass);
        a.ub_out[c * P + g] = out;
        a.w_out[c * P + g] = fma(a.a, wn, (c < 3 ? cH : cE) * out);
      }
      a.deps[g] = fma(mass, bm, d0);
    }
    __syncthreads();  // the element's shared data is consumed
  }
}

// J = sum jw |E|^2 (one partial sum per block, kSeedBlocks of them), and the
// seed ub = (0, 2 jw E), w = bdt * (hbm1 | ebm1) * ub
constexpr int kSeedThreads = 256;
__global__ void __launch_bounds__(kSeedThreads)
    k_adjoint_seed(double* w, double* ub, const double* u, const double* jw, const double* ebm1, long P,
                   double bdt, double* partial) {
  __shared__ double s_sum[kSeedThreads];
  double sum = 0.0;
  for (long g = blockIdx.x * (long)kSeedThreads + threadIdx.x; g < P; g += (long)gridDim.x * kSeedThreads) {
    const double j = jw[g], ce = bdt * ebm1[g];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double e = u[(3 + c) * P + g];
      sum = fma(j * e, e, sum);
      const double b = 2.0 * j * e;
      ub[c * P + g] = 0.0;
      w[c * P + g] = 0.0;
      ub[(3 + c) * P + g] = b;
      w[(3 + c) * P + g] = ce * b;
    }
  }
  s_sum[threadIdx.x] = sum;
  __syncthreads();
  for (int h = kSeedThreads / 2; h > 0; h /= 2) {
    if ((int)threadIdx.x < h) s_sum[threadIdx.x] += s_sum[threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = s_sum[0];
}

template <int NX, bool WIDE>
int launch_adjoint(Context* c, const AdjointDev& a) {
  using C = ACfg<NX, WIDE>;
  auto kern = k_adjoint_stage<NX, WIDE>;
  static bool ready = false;
  static int grid = 0;
  if (!ready) {
    if (check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)C::smem)))
      return NEKGPU_ERR_CUDA;
    int per_sm = 0, sms = 0;
    if (check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, C::NT, C::smem)))
      return NEKGPU_ERR_CUDA;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device);
    if (per_sm < 1) return NEKGPU_ERR_UNSUPPORTED;
    grid = per_sm * sms;
    ready = true;
  }
  const int g = c->nelt < grid ? c->nelt : grid;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(g);
  cfg.blockDim = dim3(C::NT);
  cfg.dynamicSmemBytes = C::smem;
  cfg.stream = c->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (check_cuda(cudaLaunchKernelEx(&cfg, kern, a))) return NEKGPU_ERR_CUDA;
  c->last_launches += 1;
  return check_cuda(cudaGetLastError());
}


// Wide blocks take one turn where the others take two or three, which a stage
// of few elements waits for: up to one element per SM, at N=5 three, at N <= 4
// always.  us per reverse stage with the recomputation in mixed stages, wide /
// not (a thread per node and contraction before: last): N=7 8 elements 15.1 /
// 18.8 (19.4), 64 15.9 / 21.5 (20.2), 152 22.0 / 28.9 (25.9), 300 39.8 / 41.1
// (43.5), 336 46.8 / 43.3 (53.2); N=6 64 15.9 / 20.1 (17.1), 336 38.6 / 34.0
// (41.2); N=5 64 11.5 / 16.1 (14.1), 336 23.2 / 26.4 (28.8), 608 34.0 / 34.2
// (40.0), 700 40.6 / 36.0 (47.4); N=4 64 11.3 / 13.3 (14.0), 2000 66.5 / 72.0
// (85.3).
template <int NX>
int dispatch_adjoint(Context* c, const AdjointDev& a) {
  if constexpr (NX <= 5) {
    return launch_adjoint<NX, true>(c, a);
  } else {
    return c->nelt <= (NX == 6 ? 3 : 1) * num_sms(c) ? launch_adjoint<NX, true>(c, a)
                                                     : launch_adjoint<NX, false>(c, a);
  }
}

}  // namespace

int adjoint_stage(Context* c, const AdjointDev& a) {
  switch (c->nx) {
    case 3: return dispatch_adjoint<3>(c, a);
    case 4: return dispatch_adjoint<4>(c, a);
    case 5: return dispatch_adjoint<5>(c, a);
    case 6: return dispatch_adjoint<6>(c, a);
    case 7: return dispatch_adjoint<7>(c, a);
    case 8: return dispatch_adjoint<8>(c, a);
    case 9: return dispatch_adjoint<9>(c, a);
    default: return NEKGPU_ERR_UNSUPPORTED;
  }
}

int adjoint_seed(Context* c, double* w, double* ub, const double* u, const double* jw, double bdt,
                 double* partial) {
  k_adjoint_seed<<<kSeedBlocks, kSeedThreads, 0, c->stream>>>(w, ub, u, jw, c->d_ebm1, c->npts, bdt,
                                                              partial);
  c->last_launches += 1;
  return check_cuda(cudaGetLastError());
}

}  // namespace nekgpu
