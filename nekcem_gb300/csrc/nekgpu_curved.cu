// Fused FP64 stage on curvilinear hexahedra (NEKGPU_FUSED64 on a mesh whose
// metrics vary inside the elements): the general weighted curl with all nine
// per-node metrics (maxwell_wght_curl, src/cem_maxwell.F:1428-1497), the
// upwind flux with per-face-node normals and areas and the partner's values
// read directly (cem_maxwell_flux3d and gs_op_fields,
// src/cem_maxwell.F:922-1002, 1368-1426), the lift (:725-735), the volume
// source, the inverse mass and the low-storage RK update
// (src/cem_common.F:18-75), one kernel per stage.  With the dealiased curl
// (param(18) = -1, maxwell_wght_dcurl) its volume term comes from k_dcurl,
// launched before the stage kernel, which then adds flux, lift, source,
// inverse mass and RK update in one pass.
//
// What bounds it: the FP64 pipe (two lanes per clock and SM).  The 18
// contractions per node run in 64-bit integer arithmetic (nekgpu_fixed.cuh),
// one thread per GLL line; the node's weight w3 multiplies the curl once, as
// the lift is added, and the areas are inside the face coefficients.  That
// leaves 117 FP64-pipe instructions per node at N=5 with two media (curl 36,
// flux about 60 on the many face nodes of this order, finish 18) of the ~230 of
// a form with FP64 contractions: 58.6 us per stage for 990 elements (135 before;
// FP64 pipe 77 % busy), at N=7 116 us for 1000 elements.
//
// One block per element at a time, thread per node: state in shared memory;
// face nodes' fluxes summed per node, axis by axis so that no two threads
// meet at one; then for each direction the six derivatives to
// shared memory and, per node, their products with the direction's three
// metrics into the residual held in registers.  The metrics add 72 bytes per
// node and stage to the affine kernel's traffic; the face geometry 4 doubles
// and the partner index per face node.
#include <cuda_runtime.h>

#include <algorithm>

#include "nekgpu_internal.h"
#include "nekgpu_lines.cuh"

namespace nekgpu {

namespace {

template <int NX>
__device__ __forceinline__ void face_node(int f, int a, int b, int& i, int& j, int& k) {
  // slot order s=-1, r=+1, s=+1, r=-1, t=-1, t=+1 (pff)
  const int ax = slot_axis(f), fix = slot_side(f) < 0 ? 0 : NX - 1;
  i = ax == 0 ? fix : a;
  j = ax == 1 ? fix : (ax == 0 ? a : b);
  k = ax == 2 ? fix : b;
}

template <int NX>
struct KCfg {
  static constexpr int N2 = NX * NX, N3 = N2 * NX, NF = 6 * N2;
  static constexpr int RS = NX | 1, SZ = RS * NX, N3P = NX * SZ;  // odd rows
  static constexpr int NT = round32(N3 > 6 * N2 ? N3 : 6 * N2);  // a thread per node, line and face node
  static constexpr int kMinBlocks = NT > 256 ? 2 : (NT > 160 ? 3 : 4);
  static constexpr size_t smem = 4 * 6 * (size_t)N3P * 8;  // state, derivatives A and B, lifted flux
};

// the six derivatives along DIR to s_d: one thread per (component, line)
template <int NX, int DIR>
__device__ __forceinline__ void curved_lines(const double* s_u, double* s_d, const CurvedDev& a) {
  using C = KCfg<NX>;
  const int task = threadIdx.x;
  if (task >= 6 * C::N2) return;
  const int c = task / C::N2, lam = task - c * C::N2, la = lam % NX, lb = lam / NX;
  const int base = c * C::N3P + (DIR == 0 ? C::RS * la + C::SZ * lb
                                          : (DIR == 1 ? la + C::SZ * lb : la + C::RS * lb));
  constexpr int step = DIR == 0 ? 1 : (DIR == 1 ? C::RS : C::SZ);
  line_outputs<NX, false>(s_u + base, step, 0, NX, a.fd, a.D, nullptr,
                          [&](int i, double x) { s_d[base + step * i] = x; });
}

template <int NX>
__global__ void __launch_bounds__(KCfg<NX>::NT, KCfg<NX>::kMinBlocks)
    k_curved_stage(const __grid_constant__ CurvedDev a) {
  using C = KCfg<NX>;
  constexpr int N2 = C::N2, N3 = C::N3, NF = C::NF, N3P = C::N3P;
  extern __shared__ __align__(16) unsigned char smem[];
  double* s_u = reinterpret_cast<double*>(smem);
  double* s_A = s_u + 6 * N3P;
  double* s_B = s_A + 6 * N3P;
  double* s_L = s_B + 6 * N3P;
  const int tid = threadIdx.x;
  const long P = a.npts;
  const bool node = tid < N3;
  const int vi = tid % NX, vj = (tid / NX) % NX, vk = tid / N2;
  const int pn = vi + C::RS * vj + C::SZ * vk;  // stored node
  const bool on_face = node && (vi == 0 || vi == NX - 1 || vj == 0 || vj == NX - 1 || vk == 0 || vk == NX - 1);
  const bool first_stage = (a.a == 0.0);

  // a programmatic dependent of the previous launch: nothing it wrote is read
  // before it has completed; the next one may launch from the last element on
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  for (int e = blockIdx.x; e < a.nelt; e += gridDim.x) {
    if (e + (int)gridDim.x >= a.nelt) asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    const long g = (long)e * N3 + tid;
    if (node) {
#pragma unroll
      for (int c = 0; c < 6; ++c) {
        s_u[c * N3P + pn] = a.u_in[c * P + g];
      }
    }
    // ---- upwind flux of the thread's face node, lifted -------------------------
    double F[6];
    int fax = -1, fv = 0;
    bool later = false;  // the node lies on a face of an axis before this one
    __syncthreads();
    if (tid < NF) {
      const int f = tid / N2, ab = tid - f * N2;
      int i, j, k;
      face_node<NX>(f, ab % NX, ab / NX, i, j, k);
      fv = i + C::RS * j + C::SZ * k;
      fax = slot_axis(f);
      later = (fax > 0 && (i == 0 || i == NX - 1)) || (fax > 1 && (j == 0 || j == NX - 1));
      const long js = (long)e * NF + tid, L = a.nxzfl;
      const int pv = a.partner[js];
      const double nx = a.face[js], ny = a.face[L + js], nz = a.face[2 * L + js];
      double dH[3], dE[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double em = s_u[(c + 3) * N3P + fv];
        if (pv >= 0) {
          dH[c] = a.u_in[c * P + pv] - s_u[c * N3P + fv];
          dE[c] = a.u_in[(c + 3) * P + pv] - em;
        } else {  // PEC mirror: H+ = H-, E+ = -E-
          dH[c] = 0.0;
          dE[c] = -2.0 * em;
        }
      }
      // n x [E], n x [H] (the gs sums of -n x E, -n x H) and the upwind terms
      // n x (n x [u]); the area is in the coefficients
      const double n[3] = {nx, ny, nz};
      double xE[3], xH[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const int p = (c + 1) % 3, q = (c + 2) % 3;
        xE[c] = fma(n[p], dE[q], -(n[q] * dE[p]));
        xH[c] = fma(n[p], dH[q], -(n[q] * dH[p]));
      }
      if (a.fcoef) {
        const double Y02 = a.fcoef[js], C02Y = a.fcoef[L + js], Z02 = a.fcoef[2 * L + js],
                     C02Z = a.fcoef[3 * L + js];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const int p = (c + 1) % 3, q = (c + 2) % 3;
          F[c] = fma(Y02, xE[c], -(C02Y * fma(n[p], xH[q], -(n[q] * xH[p]))));
          F[3 + c] = fma(Z02, xH[c], -(C02Z * fma(n[p], xE[q], -(n[q] * xE[p]))));
        }
      } else {  // Y02 = -1/2, C02Y = Z02 = C02Z = 1/2 times the area
        const double h = a.face[3 * L + js];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const int p = (c + 1) % 3, q = (c + 2) % 3;
          F[c] = -h * fma(n[p], xH[q], fma(-n[q], xH[p], xE[c]));
          F[3 + c] = h * fma(-n[p], xE[q], fma(n[q], xE[p], xH[c]));
        }
      }
    }
    // ---- lift, and the weighted curl resE += W curl H, resH -= W curl E ---------
    // d/dx_ax = sum over directions of metric(dir, ax) d/d_dir.  The lines of
    // one direction run beside the lift of one axis (its two faces share no
    // node) and the products of the direction before:
    //   lines r -> A, lift r | lines s -> B, lift s, A | lines t -> A, lift t, B | A
    double res[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    auto lift = [&](int ax) {
      if (fax == ax)
#pragma unroll
        for (int c = 0; c < 6; ++c) {
          double* q = s_L + c * N3P + fv;
          *q = ax > 0 && later ? *q + F[c] : F[c];
        }
    };
    auto products = [&](int dir, const double* s_d) {
      if (!node) return;
      double m[3];
#pragma unroll
      for (int ax = 0; ax < 3; ++ax) m[ax] = a.metrics[(3 * dir + ax) * P + g];
#pragma unroll
      for (int q = 0; q < 3; ++q) {  // a component enters the curl's two others
        const int p1 = (q + 1) % 3, p2 = (q + 2) % 3;
        const double h = s_d[q * N3P + pn], v = s_d[(3 + q) * N3P + pn];
        res[3 + p2] = fma(-m[p1], h, res[3 + p2]);
        res[3 + p1] = fma(m[p2], h, res[3 + p1]);
        res[p2] = fma(m[p1], v, res[p2]);
        res[p1] = fma(-m[p2], v, res[p1]);
      }
    };
    const bool curl = a.vres == nullptr;  // else the dealiased volume term, computed before
    lift(0);
    if (curl) curved_lines<NX, 0>(s_u, s_A, a);
    __syncthreads();
    lift(1);
    if (curl) {
      curved_lines<NX, 1>(s_u, s_B, a);
      products(0, s_A);
    }
    __syncthreads();
    lift(2);
    if (curl) {
      curved_lines<NX, 2>(s_u, s_A, a);
      products(1, s_B);
    }
    __syncthreads();
    if (curl) {
      products(2, s_A);
      const double w3 = node ? a.w3[tid] : 0.0;
#pragma unroll
      for (int c = 0; c < 6; ++c) res[c] = fma(w3, res[c], on_face ? s_L[c * N3P + pn] : 0.0);
    } else if (node) {
#pragma unroll
      for (int c = 0; c < 6; ++c) res[c] = a.vres[c * P + g] + (on_face ? s_L[c * N3P + pn] : 0.0);
    }
    if (node) {
      // ---- volume source (usersrc) ---------------------------------------
      if (a.src_elem) {
        const int so = a.src_elem[e];
        if (so >= 0) res[5] = fma(a.src_w[(long)so * N3 + tid], a.src_ft, res[5]);
      }
      // ---- inverse mass + low-storage RK ---------------------------------
      const double ch = a.coef[g], ce = a.coef[P + g];
      double kk[6];
#pragma unroll
      for (int c = 0; c < 6; ++c) kk[c] = first_stage ? 0.0 : a.k[c * P + g];
#pragma unroll
      for (int c = 0; c < 6; ++c) {
        const double r = res[c] * (c < 3 ? ch : ce);
        const double kn = first_stage ? r : fma(a.a, kk[c], r);
        a.k[c * P + g] = kn;
        a.u_out[c * P + g] = fma(a.b, kn, s_u[c * N3P + pn]);
      }
    }
    // (the next element's state overwrites s_u: only this thread's node of it
    // is still read above)
  }
}

template <int NX>
int launch_curved(Context* c, const CurvedDev& a) {
  using C = KCfg<NX>;
  static int grid = 0;
  if (!grid) {
    if (check_cuda(cudaFuncSetAttribute(k_curved_stage<NX>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)C::smem)))
      return NEKGPU_ERR_CUDA;
    int per_sm = 0;
    if (check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_curved_stage<NX>, C::NT,
                                                                 C::smem)))
      return NEKGPU_ERR_CUDA;
    if (per_sm < 1) return NEKGPU_ERR_UNSUPPORTED;
    grid = per_sm * num_sms(c);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(std::min(c->nelt, grid));
  cfg.blockDim = dim3(C::NT);
  cfg.dynamicSmemBytes = C::smem;
  cfg.stream = c->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (check_cuda(cudaLaunchKernelEx(&cfg, k_curved_stage<NX>, a))) return NEKGPU_ERR_CUDA;
  c->last_launches += 1;
  return check_cuda(cudaGetLastError());
}

}  // namespace

int curved_stage(Context* c, int rkstep, double time, double dt) {
  int st = scale_coef(c, dt);
  if (st) return st;
  CurvedDev a = c->cargs;
  a.u_in = c->d_u[c->cur];
  a.u_out = c->d_u[c->cur ^ 1];
  a.a = c->rk_a[rkstep - 1];
  a.b = c->rk_b[rkstep - 1];
  a.src_elem = c->fargs.src_elem;
  a.src_w = reinterpret_cast<const double*>(c->fargs.src_w);
  if (c->src.enabled) a.src_ft = source_ft(c->src, time + dt * c->rk_c[rkstep - 1]);
  a.vres = nullptr;
  if (c->pargs.md > 0) {  // param(18) = -1: the dealiased curl of the stage's input
    if ((st = dcurl_into(c, a.u_in, c->d_vres))) return st;
    a.vres = c->d_vres;
  }
  switch (c->nx) {
    case 3: st = launch_curved<3>(c, a); break;
    case 4: st = launch_curved<4>(c, a); break;
    case 5: st = launch_curved<5>(c, a); break;
    case 6: st = launch_curved<6>(c, a); break;
    case 7: st = launch_curved<7>(c, a); break;
    case 8: st = launch_curved<8>(c, a); break;
    default: return NEKGPU_ERR_UNSUPPORTED;
  }
  if (st) return st;
  c->cur ^= 1;
  return NEKGPU_OK;
}

}  // namespace nekgpu
