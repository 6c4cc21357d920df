// Fused FP64 stage on affine axis-aligned hexahedra (NEKGPU_FUSED64): weighted
// curl (src/nek5_grad.F:2-19, src/cem_maxwell.F:1428-1497), upwind face flux
// with the in-kernel partner read that replaces gs_op_fields
// (src/cem_maxwell.F:922-1002, 1368-1426), lift (src/cem_maxwell.F:725-735),
// PML, dispersive currents, incident fields, graphene sheets, volume source,
// inverse mass (src/cem_maxwell.F:1878-1886) and the low-storage RK update
// (src/cem_common.F:18-75), one kernel per stage.
//
// What bounds it: GB300 issues two FP64 lanes per clock and SM.  With the
// contractions in FP64 (96 of its 206 FP64-pipe instructions per node at N=7) a
// stage of the 16^3-element N=7 box took 690 us; it takes 221 us (57 G DOF-stage
// updates/s, FP64 pipe 61 % busy) with
//  * the contractions in 64-bit integer arithmetic (nekgpu_fixed.cuh) on
//    another pipe, one thread per GLL line, D as constant-bank operands;
//  * the residual normalised by w3*rx as in the mixed form, so that the curl
//    takes one FP64 multiply-add per derivative at most (none for the r-lines),
//    the lift factor is part of the face coefficients, and w3 is folded into
//    the inverse-mass coefficient;
//  * only the four field components tangential to a face in its flux.
// 40.5 FP64-pipe instructions per node are left (finish 18, curl 8, flux 12): 20
// of the 33 clocks per node and SM.
//
// Phases per element: state to shared memory (8-byte asynchronous copies into
// an odd row length), flux per face node, two phases of line tasks into the
// residual, then node by node the finish.  The split form gives an element's
// k-slabs to several blocks, for meshes with fewer elements than SMs: every
// block stages the whole element (the t-lines need it) and works out the
// nodes of its slab, so the blocks share nothing.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "nekgpu_internal.h"
#include "nekgpu_lines.cuh"

namespace nekgpu {

namespace {

template <int NX>
struct DCfg : ElemCfg<NX> {
  using E = ElemCfg<NX>;
  // state, residual, flux [face][line slot][N2], D rows (split form)
  static constexpr size_t off_R = 6 * (size_t)E::N3P * 8, off_F = 2 * off_R;
  static constexpr size_t off_D = (off_F + 24 * (size_t)E::N2 * 8 + 15) / 16 * 16;
  static constexpr size_t smem(bool split) { return off_D + (split ? E::N2 * 8 : 0); }
};

// The part of an element a block works out: its nodes with k in [k0, k1).
struct Slab {
  int k0, k1;
};

// Face task t of the slab: slot f and in-face node (a, b)
template <int NX, bool SPLIT>
__device__ __forceinline__ int face_tasks(Slab s) {
  if (!SPLIT) return 6 * NX * NX;
  return 4 * NX * (s.k1 - s.k0) + (s.k0 == 0 ? NX * NX : 0) + (s.k1 == NX ? NX * NX : 0);
}
template <int NX, bool SPLIT>
__device__ __forceinline__ void face_task(Slab s, int t, int& f, int& a, int& b) {
  constexpr int N2 = NX * NX;
  if (!SPLIT) {
    f = t / N2;
    a = t % NX;
    b = (t - f * N2) / NX;
    return;
  }
  const int per = NX * (s.k1 - s.k0);
  if (t < 4 * per) {  // the side faces: rows b = k of the slab
    f = t / per;
    const int ab = t - f * per;
    a = ab % NX;
    b = s.k0 + ab / NX;
    return;
  }
  t -= 4 * per;
  f = s.k0 == 0 && t < N2 ? 4 : 5;
  if (f == 5 && s.k0 == 0) t -= N2;
  a = t % NX;
  b = t / NX;
}

// One output x of a line task into the residual: the r-lines (OP 0) start
// their components, whose derivative has coefficient one; the s-lines of
// phase 0 (OP 1) start theirs times rho; phase 1 (OP 2) completes all six.  F
// is the lifted flux at a line's end.
template <int OP>
__device__ __forceinline__ void line_put(double* Rp, double x, bool neg, double rho, bool end, double F) {
  double v;
  if (OP == 0) {
    v = flip(x, neg);
    if (end) v += F;
  } else if (OP == 1) {
    v = fma(flip(rho, neg), x, end ? F : 0.0);
  } else {
    v = fma(flip(rho, neg), x, *Rp);
    if (end) v += F;
  }
  *Rp = v;
}

// Line type `type` of phase PH along line lam: outputs [i0, i1) (all of them
// unless SPLIT, which takes D's rows from shared memory instead of the
// constant bank).
template <int NX, int PH, int OP, bool SPLIT>
__device__ __forceinline__ void line_task(int type, int lam, int i0, int i1, const double* s_u,
                                          double* s_R, const double* s_F, const int2* s_D,
                                          double rho_s, double rho_t, const Fp64Dev& a) {
  using C = DCfg<NX>;
  constexpr int N2 = C::N2;
  const LineType& lt = kLine[PH][type];
  const int dir = lt.dir;
  const bool neg = lt.neg != 0;
  const int la = lam % NX, lb = lam / NX;
  const int base = dir == 0 ? C::RS * la + C::SZ * lb : (dir == 1 ? la + C::SZ * lb : la + C::RS * lb);
  const int step = dir == 0 ? 1 : (dir == 1 ? C::RS : C::SZ);
  const double rho = dir == 2 ? rho_t : rho_s;
  const double* pu = s_u + lt.comp * C::N3P + base;
  double* R = s_R + lt.res * C::N3P + base;
  // faces 3|1 (r), 0|2 (s), 4|5 (t)
  const double* Fm = s_F + ((dir == 0 ? 3 : (dir == 1 ? 0 : 4)) * 4 + lt.slot) * N2 + lam;
  const double* Fp = s_F + ((dir == 0 ? 1 : (dir == 1 ? 2 : 5)) * 4 + lt.slot) * N2 + lam;
  line_outputs<NX, SPLIT>(pu, step, i0, i1, a.fd, a.D, s_D, [&](int i, double x) {
    const bool end = i == 0 || i == NX - 1;
    line_put<OP>(R + step * i, x, neg, rho, end, end ? (i == 0 ? *Fm : *Fp) : 0.0);
  });
}

// Phase PH of the contractions over the slab: tasks (line type, line), in the
// split form (type, group of og outputs, line).
template <int NX, int PH, bool SPLIT>
__device__ __forceinline__ void line_phase(const double* s_u, double* s_R, const double* s_F,
                                           const int2* s_D, double rho_s, double rho_t, Slab sl,
                                           int og, const Fp64Dev& a) {
  using C = DCfg<NX>;
  constexpr int N2 = C::N2, NT = C::NT;
  const int tid = threadIdx.x;
  if constexpr (!SPLIT) {
    constexpr int NA = PH == 0 ? 4 : 6;  // types of the phase's first operation
#pragma unroll 1
    for (int task = tid; task < NA * N2; task += NT) {
      const int type = task / N2;
      line_task<NX, PH, PH == 0 ? 0 : 2, false>(type, task - type * N2, 0, NX, s_u, s_R, s_F, s_D,
                                                rho_s, rho_t, a);
    }
    if (PH == 0) {
      // the other two types, starting with the threads the first four left idle
      constexpr int off = (NA * N2) % NT;
#pragma unroll 1
      for (int task = tid >= off ? tid - off : tid + NT - off; task < 2 * N2; task += NT) {
        const int type = task / N2;
        line_task<NX, 0, 1, false>(NA + type, task - type * N2, 0, NX, s_u, s_R, s_F, s_D, rho_s,
                                   rho_t, a);
      }
    }
  } else {
    // r and s types run along the slab's lines, t types along all lines
    const int nl = NX * (sl.k1 - sl.k0), nrs = nl * ((NX + og - 1) / og);
    const int nt = N2 * ((sl.k1 - sl.k0 + og - 1) / og);
    const int nrt = PH == 0 ? 6 : 2;
    const int ntask = nrt * nrs + (6 - nrt) * nt;
#pragma unroll 1
    for (int task = tid; task < ntask; task += NT) {
      if (PH == 0 || task < 2 * nrs) {
        const int type = task / nrs, q = task - type * nrs, grp = q / nl;
        const int lam = q - grp * nl + NX * sl.k0, i0 = grp * og, i1 = min(NX, i0 + og);
        if (PH == 0 && type < 4)
          line_task<NX, 0, 0, true>(type, lam, i0, i1, s_u, s_R, s_F, s_D, rho_s, rho_t, a);
        else
          line_task<NX, PH, PH == 0 ? 1 : 2, true>(type, lam, i0, i1, s_u, s_R, s_F, s_D, rho_s, rho_t, a);
      } else {
        const int q0 = task - 2 * nrs, type = q0 / nt, q = q0 - type * nt, grp = q / N2;
        const int i0 = sl.k0 + grp * og, i1 = min(sl.k1, i0 + og);
        line_task<NX, 1, 2, true>(2 + type, q - grp * N2, i0, i1, s_u, s_R, s_F, s_D, rho_s, rho_t, a);
      }
    }
  }
}

// PML (pml_step, src/cem_maxwell_pml.F:508-590) at one node of a PML element:
// the auxiliary fields' RK update (src/cem_maxwell.F:1942-1955) and the PML
// terms added to R; the coefficients are those of PmlDev (seven FP64
// operations per component; ten from sigma, mu and bm1).
template <int N3>
__device__ __forceinline__ void pml_node(const Fp64Dev& a, int l, int v, const double* u,
                                         bool first_stage, double* R) {
  const long nn = a.pml.n, q = (long)l * N3 + v;
  const double* pd = a.pml.data + q;
  double* aux = a.pml.aux + q;
  double* kx = a.pml.k + q;
  // every load before the stores, which they could not pass
  const double fac = __ldg(pd + 12 * nn);
  double f[6], kk[6], s1[3], A[3], B[6];
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    f[c] = aux[c * nn];
    kk[c] = first_stage ? 0.0 : kx[c * nn];
    B[c] = __ldg(pd + (6 + c) * nn);
    if (c < 3) {
      s1[c] = __ldg(pd + c * nn);
      A[c] = __ldg(pd + (3 + c) * nn);
    }
  }
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    const int d = c % 3;
    const double rp = fma(R[c], fac, -(s1[d] * f[c]));
    const double kv = first_stage ? a.dt * rp : fma(a.a, kk[c], a.dt * rp);
    R[c] = fma(A[d], f[c], fma(-B[c], u[c], R[c]));
    kx[c * nn] = kv;
    aux[c * nn] = fma(a.b, kv, f[c]);
  }
}

// Dispersive currents inside usersrc (cem_maxwell_drude / cem_maxwell_lorentz,
// src/cem_maxwell.F:3095-3212): resE -= J1 bm1, the currents' RK update.
template <int N3>
__device__ __forceinline__ void disp_node(const Fp64Dev& a, int l, int v, const double* u,
                                          bool first_stage, double* R) {
  const DispDev& d = a.disp;
  const long nn = d.n, q = (long)l * N3 + v;
  const int kind = (int)d.data[q];
  if (kind == 0) return;
  const double pa = d.data[nn + q], pb = d.data[2 * nn + q], pc = d.data[3 * nn + q];
  const double inv = d.data[5 * nn + q];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double j1 = d.aux[c * nn + q], ev = u[3 + c];
    R[3 + c] -= j1 * inv;
    double r1 = -pa * j1 + pb * ev;
    if (kind == 2) {
      const double j2 = d.aux[(3 + c) * nn + q];
      r1 = -pa * j1 - pb * j2 + pc * ev;
      const double k2 = first_stage ? a.dt * j1 : fma(a.a, d.k[(3 + c) * nn + q], a.dt * j1);
      d.k[(3 + c) * nn + q] = k2;
      d.aux[(3 + c) * nn + q] = fma(a.b, k2, j2);
    }
    const double k1 = first_stage ? a.dt * r1 : fma(a.a, d.k[c * nn + q], a.dt * r1);
    d.k[c * nn + q] = k1;
    d.aux[c * nn + q] = fma(a.b, k1, j1);
  }
}

// Graphene sheet (userfsrc) at a face node of slot f: n x J with the currents J
// of the own (go) and the partner's (gp) listed slot, which the sheet adds to
// [H] (n x [H] - J), from the fields h, ev here and hp, ep there (the incident
// field included).  A PEC face keeps its mirror flux.
__device__ __noinline__ double3 sheet_jump(const Fp64Dev& a, int f, int pe, int go, int gp, double3 h,
                                           double3 ev, double3 hp, double3 ep, bool first_stage) {
  double nv[3], nm[3], J[3] = {0.0, 0.0, 0.0};
  const double hm[3] = {h.x, h.y, h.z}, em[3] = {ev.x, ev.y, ev.z};
  const double hq[3] = {hp.x, hp.y, hp.z}, eq[3] = {ep.x, ep.y, ep.z};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    nv[c] = c == slot_axis(f) ? (double)slot_side(f) : 0.0;
    nm[c] = -nv[c];
  }
  if (go >= 0) graphene_slot(a.gr, go, nv, hm, em, true, first_stage, a.a, a.b, a.dt, J);
  if (gp >= 0 && pe >= 0) graphene_slot(a.gr, gp, nm, hq, eq, false, first_stage, a.a, a.b, a.dt, J);
  if (pe < 0) return make_double3(0.0, 0.0, 0.0);
  return make_double3(nv[1] * J[2] - nv[2] * J[1], nv[2] * J[0] - nv[0] * J[2],
                      nv[0] * J[1] - nv[1] * J[0]);
}

// Blocks per SM the launch is built for.  EXT 1 at N=4: four blocks of 128
// threads (128 registers; built for two the compiler takes 204: 336 elements
// with PML 25.5 us per stage with 96 threads, 19.8 built for four, 18.4 with 128
// threads; 1000 elements 50.4, 32.0, 29.0).
template <int NX, int EXT>
constexpr int fp64_min_blocks() {
  return EXT == 1 && NX == 5 ? 4 : (NX == 9 || EXT ? 2 : (NX == 8 ? 3 : 4));
}

template <int NX, int EXT, bool SPLIT>
__global__ void __launch_bounds__(DCfg<NX>::NT, fp64_min_blocks<NX, EXT>())
    k_fp64_stage(const __grid_constant__ Fp64Dev a, int nsplit, int og) {
  using C = DCfg<NX>;
  constexpr int N2 = C::N2, N3 = C::N3, NT = C::NT, NF = C::NF;
  constexpr int NPC = EXT == 2 ? 6 : 4;
  extern __shared__ __align__(16) unsigned char smem[];
  double* s_u = reinterpret_cast<double*>(smem);
  double* s_R = reinterpret_cast<double*>(smem + C::off_R);
  double* s_F = reinterpret_cast<double*>(smem + C::off_F);
  int2* s_D = reinterpret_cast<int2*>(smem + C::off_D);
  const int tid = threadIdx.x;
  const long P = a.npts;
  const bool first_stage = (a.a == 0.0);  // rk4a(1) = 0: k restarts
  if (SPLIT)
    for (int t = tid; t < N2; t += NT) s_D[t] = make_int2(a.fd.hi[t], a.fd.lo[t]);
  // a programmatic dependent of the previous stage: nothing it wrote is read
  // before it has completed; the next stage may launch from the last task on
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  const int ntask = SPLIT ? a.nelt * nsplit : a.nelt;
  for (int w = blockIdx.x; w < ntask; w += gridDim.x) {
    if (w + (int)gridDim.x >= ntask) asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    const int q0 = SPLIT ? w / nsplit : w;
    const int e = EXT == 1 && a.pml.order ? a.pml.order[q0] : q0;  // (see PmlDev::order)
    Slab sl{0, NX};
    if (SPLIT) {
      const int q = w - q0 * nsplit;
      sl = Slab{q * NX / nsplit, (q + 1) * NX / nsplit};
    }
    const int* nbr = a.nbr + 6 * (long)e;
    const double* eg = a.egn + 14 * (long)e;
    // ---- own state to shared memory, partner face values to registers --------
    for (int v = tid; v < N3; v += NT) {
      const int pv = pnode<NX>(v);
#pragma unroll
      for (int c = 0; c < 6; ++c)
        cp_async8(s_u + c * C::N3P + pv, a.u_in + c * P + (long)e * N3 + v);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    // what the finish reads, and the next element's state, on their way to L2
    if (!SPLIT) {
      const int wn = w + (int)gridDim.x;
      const int en = wn < ntask ? (EXT == 1 && a.pml.order ? a.pml.order[wn] : wn) : e;
#pragma unroll 1
      for (int t = tid; t < 14 * ((N3 + 15) / 16); t += NT) {
        const int q = t / ((N3 + 15) / 16), o = 16 * (t - q * ((N3 + 15) / 16));
        const double* p = q < 6 ? a.u_in + q * P + (long)en * N3
                                : (q < 12 ? a.k + (q - 6) * P : a.coef + (q - 12) * P) + (long)e * N3;
        asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p + o));
      }
    }
    const int nft = face_tasks<NX, SPLIT>(sl);
    double nbv[C::FPT][NPC];
#pragma unroll
    for (int q = 0; q < C::FPT; ++q) {
      const int t = tid + q * NT;
      if (t < nft) {
        int f, fa, fb;
        face_task<NX, SPLIT>(sl, t, f, fa, fb);
        const int pe = nbr[f];
        if (pe >= 0) {
          const long pv = (long)pe * N3 + face_vol<NX>(slot_opp(f), fa, fb);
#pragma unroll
          for (int k = 0; k < NPC; ++k) nbv[q][k] = __ldg(a.u_in + partner_comp<EXT>(f, k) * P + pv);
        }
      }
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    // ---- upwind flux per face node, lifted, into s_F ---------------------------
    // rows of the listed elements in the incident field's and the sheets' tables
    const int io = EXT == 2 && a.inc_elem ? a.inc_elem[e] : -1;
    const int gr = EXT == 2 && a.gr.elem ? a.gr.elem[e] : -1;
#pragma unroll
    for (int q = 0; q < C::FPT; ++q) {
      const int t = tid + q * NT;
      if (t >= nft) continue;
      int f, fa, fb;
      face_task<NX, SPLIT>(sl, t, f, fa, fb);
      const int j = f * N2 + fa + NX * fb;
      const int pv = pnode<NX>(face_vol<NX>(f, fa, fb));
      const int pe = nbr[f];
      const int ax = slot_axis(f);
      // the tangential axes ta < tb; jumps partner - own (PEC mirror: [H] = 0,
      // [E] = -2 E)
      const int ta = ax == 0 ? 1 : 0, tb = ax == 2 ? 1 : 2;
      double JHa, JHb, JEa, JEb;
      if (EXT == 2) {
        double h[3], ev[3], hp[3], ep[3], JH[3], JE[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          h[c] = s_u[c * C::N3P + pv];
          ev[c] = s_u[(3 + c) * C::N3P + pv];
          hp[c] = pe >= 0 ? nbv[q][c] : 0.0;
          ep[c] = pe >= 0 ? nbv[q][EXT == 2 ? 3 + c : 0] : 0.0;
        }
        // userinc: the incident field on the own side of a listed face node, or
        // on the partner's side when the partner's slot is listed
        if (io >= 0) {
          const double* iv = a.inc_val + (long)io * 12 * NF + j;
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            h[c] += iv[c * NF];
            ev[c] += iv[(3 + c) * NF];
            hp[c] += iv[(6 + c) * NF];
            ep[c] += iv[(9 + c) * NF];
          }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          JH[c] = pe >= 0 ? hp[c] - h[c] : 0.0;
          JE[c] = pe >= 0 ? ep[c] - ev[c] : -2.0 * ev[c];
        }
        if (gr >= 0) {
          const int go = a.gr.own[(long)gr * NF + j], gp = a.gr.part[(long)gr * NF + j];
          if (go >= 0 || gp >= 0) {
            const double3 d = sheet_jump(a, f, pe, go, gp, make_double3(h[0], h[1], h[2]),
                                         make_double3(ev[0], ev[1], ev[2]), make_double3(hp[0], hp[1], hp[2]),
                                         make_double3(ep[0], ep[1], ep[2]), first_stage);
            JH[0] += d.x;
            JH[1] += d.y;
            JH[2] += d.z;
          }
        }
        JHa = ax == 0 ? JH[1] : JH[0];
        JHb = ax == 2 ? JH[1] : JH[2];
        JEa = ax == 0 ? JE[1] : JE[0];
        JEb = ax == 2 ? JE[1] : JE[2];
      } else {
        const double ea = s_u[(3 + ta) * C::N3P + pv], eb = s_u[(3 + tb) * C::N3P + pv];
        if (pe >= 0) {
          JHa = nbv[q][0] - s_u[ta * C::N3P + pv];
          JHb = nbv[q][1] - s_u[tb * C::N3P + pv];
          JEa = nbv[q][2] - ea;
          JEb = nbv[q][3] - eb;
        } else {
          JHa = JHb = 0.0;
          JEa = -2.0 * ea;
          JEb = -2.0 * eb;
        }
      }
      // In the line slot order of the face's direction (residuals 5,4,2,1 |
      // 5,3,2,0 | 4,3,1,0), with s = side for faces normal to r and t, -side
      // for s:  F0 = s Z JHa + CZ JEb,  F1 = -s Z JHb + CZ JEa,
      //         F2 = s Y JEa + CY JHb,  F3 = -s Y JEb + CY JHa,
      // the coefficients times the lift factor (uniform media: Y = -1/2,
      // Z = 1/2, CY = CZ = C0/2).
      const bool neg = (slot_side(f) < 0) != (ax == 1);
      double2 cy, cz;
      if (a.fcoef) {
        const double2* fc = reinterpret_cast<const double2*>(a.fcoef + 4 * ((long)e * NF + j));
        cy = fc[0];
        cz = fc[1];
      } else {
        cz = make_double2(eg[2 + f], eg[8 + f]);
        cy = make_double2(flip(cz.x, true), cz.y);
      }
      double* Fo = s_F + f * 4 * N2 + fa + NX * fb;
      Fo[0] = fma(cz.x, flip(JHa, neg), cz.y * JEb);
      Fo[N2] = fma(cz.x, flip(JHb, !neg), cz.y * JEa);
      Fo[2 * N2] = fma(cy.x, flip(JEa, neg), cy.y * JHb);
      Fo[3 * N2] = fma(cy.x, flip(JEb, !neg), cy.y * JHa);
    }
    __syncthreads();
    const double rho_s = eg[0], rho_t = eg[1];
    line_phase<NX, 0, SPLIT>(s_u, s_R, s_F, s_D, rho_s, rho_t, sl, og, a);
    __syncthreads();
    line_phase<NX, 1, SPLIT>(s_u, s_R, s_F, s_D, rho_s, rho_t, sl, og, a);
    __syncthreads();
    // ---- PML, currents, source, inverse mass, RK update, node by node ----------
    const int so = a.src_elem ? a.src_elem[e] : -1;
    const int pml_l = (EXT > 0 && a.pml.slot) ? a.pml.slot[e] : -1;
    const int disp_l = (EXT > 0 && a.disp.slot) ? a.disp.slot[e] : -1;
#pragma unroll 1
    for (int v = tid + sl.k0 * N2; v < sl.k1 * N2; v += NT) {
      const int pv = pnode<NX>(v);
      const long g = (long)e * N3 + v;
      double R[6], u[6], kk[6];
#pragma unroll
      for (int c = 0; c < 6; ++c) kk[c] = first_stage ? 0.0 : a.k[c * P + g];
      const double ch = a.coef[g], ce = a.coef[P + g];
#pragma unroll
      for (int c = 0; c < 6; ++c) {
        R[c] = s_R[c * C::N3P + pv];
        u[c] = s_u[c * C::N3P + pv];
      }
      if (EXT > 0 && pml_l >= 0) pml_node<N3>(a, pml_l, v, u, first_stage, R);
      if (EXT > 0 && disp_l >= 0) disp_node<N3>(a, disp_l, v, u, first_stage, R);
      if (so >= 0) R[5] = fma(a.src_w[(long)so * N3 + v], a.src_ft, R[5]);
#pragma unroll
      for (int c = 0; c < 6; ++c) {
        const double r = R[c] * (c < 3 ? ch : ce);
        const double kn = first_stage ? r : fma(a.a, kk[c], r);
        a.k_out[c * P + g] = kn;
        a.u_out[c * P + g] = fma(a.b, kn, u[c]);
      }
    }
    if (w + (int)gridDim.x < ntask) __syncthreads();  // the element's shared data is consumed
  }
}

template <int NX, int EXT, bool SPLIT>
int launch(Context* c, const Fp64Dev& a, bool pdl, int nsplit, int og) {
  using C = DCfg<NX>;
  constexpr size_t smem = C::smem(SPLIT);
  auto kern = k_fp64_stage<NX, EXT, SPLIT>;
  static int grid = 0;
  if (!grid) {
    if (check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)))
      return NEKGPU_ERR_CUDA;
    int per_sm = 0;
    if (check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, C::NT, smem)))
      return NEKGPU_ERR_CUDA;
    if (per_sm < 1) return NEKGPU_ERR_UNSUPPORTED;
    grid = per_sm * num_sms(c);
  }
  const int n = a.nelt * nsplit, g = n < grid ? n : grid;
  c->fused_grid = g;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(g);
  cfg.blockDim = dim3(C::NT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = c->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  if (check_cuda(cudaLaunchKernelEx(&cfg, kern, a, nsplit, og))) return NEKGPU_ERR_CUDA;
  c->last_launches += 1;
  return check_cuda(cudaGetLastError());
}

// Fewer elements than half the SMs: each is split over as many blocks as give
// one block per SM (us per stage: 27 elements, N=8: 10.2 in five slabs, 11.5 in
// three or four, 17.9 unsplit; 64 elements, N=7: 11.2 in two, 12.7 in four,
// 13.4 unsplit; with PML 15.0, 14.4, 20.5).  With more elements the slabs only
// repeat the staging and the t-lines' conversions (100 elements, N=7: 13.3
// unsplit, 14.7 in two; with PML 20.5, 21.2).  N=2 is not split in two (64
// elements: 9.4, unsplit 8.3, in three 8.0); at N=3 and 4 the two are equal.
template <int NX, int EXT>
int dispatch_split(Context* c, const Fp64Dev& a, bool pdl) {
  // outputs per task of a split line: three at NX = 9 (10.0 against 10.6 us
  // with five), halves otherwise (64 elements, N=7: 10.8 us, 12.1 with three,
  // 11.4 with two)
  constexpr int og = NX == 9 ? 3 : (NX + 1) / 2;
  const int ns = std::min(num_sms(c) / a.nelt, NX);
  return ns >= (NX == 3 ? 3 : 2) ? launch<NX, EXT, true>(c, a, pdl, ns, og) : launch<NX, EXT, false>(c, a, pdl, 1, NX);
}

template <int EXT>
int dispatch(Context* c, const Fp64Dev& a, bool pdl) {
  switch (c->nx) {
    case 3: return dispatch_split<3, EXT>(c, a, pdl);
    case 4: return dispatch_split<4, EXT>(c, a, pdl);
    case 5: return dispatch_split<5, EXT>(c, a, pdl);
    case 6: return dispatch_split<6, EXT>(c, a, pdl);
    case 7: return dispatch_split<7, EXT>(c, a, pdl);
    case 8: return dispatch_split<8, EXT>(c, a, pdl);
    case 9: return dispatch_split<9, EXT>(c, a, pdl);
    default: return NEKGPU_ERR_UNSUPPORTED;
  }
}

int fp64_launch(Context* c, Fp64Dev& a, int rkstep, double time, double dt, bool pdl) {
  a.a = c->rk_a[rkstep - 1];
  a.b = c->rk_b[rkstep - 1];
  a.dt = dt;
  a.src_elem = c->fargs.src_elem;
  a.src_w = reinterpret_cast<const double*>(c->fargs.src_w);
  if (c->src.enabled) a.src_ft = source_ft(c->src, time + dt * c->rk_c[rkstep - 1]);
  if (a.inc_elem || a.gr.elem) return dispatch<2>(c, a, pdl);
  return a.pml.slot || a.disp.slot ? dispatch<1>(c, a, pdl) : dispatch<0>(c, a, pdl);
}

// line_outputs over arrays (self-test of the fixed-point contractions)
struct LinesDev {
  FixedD fd;
  double D[kMaxFixed * kMaxFixed];
};
template <int NX, bool SPLIT>
__global__ void __launch_bounds__(256) k_fixed_lines(const __grid_constant__ LinesDev a, const double* u,
                                                     double* out, long n) {
  __shared__ int2 s_D[NX * NX];
  for (int t = threadIdx.x; t < NX * NX; t += blockDim.x) s_D[t] = make_int2(a.fd.hi[t], a.fd.lo[t]);
  __syncthreads();
  const long line = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (line >= n) return;
  double* o = out + line * NX;
  line_outputs<NX, SPLIT>(u + line * NX, 1, 0, NX, a.fd, a.D, s_D, [&](int i, double x) { o[i] = x; });
}
template <int NX>
int launch_lines(const LinesDev& a, const double* u, double* out, long n, bool split) {
  const unsigned g = (unsigned)((n + 255) / 256);
  if (split) k_fixed_lines<NX, true><<<g, 256>>>(a, u, out, n);
  else k_fixed_lines<NX, false><<<g, 256>>>(a, u, out, n);
  return check_cuda(cudaGetLastError());
}

}  // namespace

// The fixed-point table of D (nekgpu_fixed.cuh): the largest scale 2^kd with
// |D| 2^kd <= 2^61 whose cross sums stay below 2^63 for any line (the first one
// tried for the GLL matrices of N=2..8; the second for N=8's weighted transpose).
void fixed_table(const double* D, int n, FixedD& t) {
  t = FixedD{};
  double dmax = 0.0;
  bool fine = n <= kMaxFixed;
  for (int k = 0; k < n * n; ++k) {
    fine = fine && std::isfinite(D[k]);
    dmax = std::fmax(dmax, std::fabs(D[k]));
  }
  if (!fine || !(dmax > 0.0)) return;
  int ex = 0;
  std::frexp(dmax, &ex);  // dmax < 2^ex
  for (int kd = 61 - ex; kd >= 55 - ex; --kd) {
    if (kd > 150 || kd < -60) return;
    bool fits = true;
    for (int i = 0; i < n && fits; ++i) {
      double cross = 0.0;  // bounds sum |h L + l H|, and sum |h H| with it
      for (int l = 0; l < n; ++l) {
        const int k = i + n * l;
        const long long m = std::llrint(std::fabs(std::ldexp(D[k], kd)));
        const long long H = (m + (1LL << 30)) >> 31, L = m - (H << 31);
        const int s = D[k] < 0 ? -1 : 1;
        t.hi[k] = s * (int)H;
        t.lo[k] = s * (int)L;
        cross += (double)(1 << 30) * ((double)H + std::fabs((double)L));
      }
      fits = cross < 9.2e18;
    }
    if (fits) {
      t.ok = 1;
      t.bias = 1021 + kd;
      // fixed_join's exponent field stays below that of infinity: the largest
      // output, 2^63 2^(E - bias), has 1023 + 63 + E - bias
      t.maxexp = std::min(kFixedMaxExp, t.bias + 960);
      return;
    }
  }
}

int fixed_lines_selftest(int nx, const double* D, const double* u, double* out, long n, bool split) {
  LinesDev a{};
  for (int k = 0; k < nx * nx; ++k) a.D[k] = D[k];
  fixed_table(a.D, nx, a.fd);
  switch (nx) {
    case 3: return launch_lines<3>(a, u, out, n, split);
    case 4: return launch_lines<4>(a, u, out, n, split);
    case 5: return launch_lines<5>(a, u, out, n, split);
    case 6: return launch_lines<6>(a, u, out, n, split);
    case 7: return launch_lines<7>(a, u, out, n, split);
    case 8: return launch_lines<8>(a, u, out, n, split);
    case 9: return launch_lines<9>(a, u, out, n, split);
    default: return NEKGPU_ERR_UNSUPPORTED;
  }
}

int fp64_stage_buffers(Context* c, int rkstep, double time, double dt, const double* u_in,
                       double* u_out, const double* k_in, double* k_out) {
  const int st = scale_coef(c, dt);
  if (st) return st;
  Fp64Dev a = c->dargs;
  a.u_in = u_in;
  a.u_out = u_out;
  a.k = k_in;
  a.k_out = k_out;
  // not a programmatic dependent: its blocks, waiting on the SMs, would take
  // the room of the reverse stages beside it (8^3 box at N=7: 36.9 against
  // 32.2 ms per 100 steps' reverse sweep)
  return fp64_launch(c, a, rkstep, time, dt, false);
}

int fp64_stage(Context* c, int rkstep, double time, double dt) {
  int st = scale_coef(c, dt);
  if (st) return st;
  Fp64Dev a = c->dargs;
  a.u_in = c->d_u[c->cur];
  a.u_out = c->d_u[c->cur ^ 1];
  a.disp = c->fargs.disp;
  a.inc_elem = c->fargs.inc_elem;
  a.inc_val = c->fargs.inc_val;
  a.gr = c->fargs.gr;
  if (a.inc_elem && (st = incident_upload(c, time + dt * c->rk_c[rkstep - 1]))) return st;
  if (a.gr.elem) {
    a.gr.f_in = c->d_gr_f[c->gr_cur];
    a.gr.f_out = c->d_gr_f[c->gr_cur ^ 1];
  }
  if ((st = fp64_launch(c, a, rkstep, time, dt, true))) return st;
  if (a.gr.elem) c->gr_cur ^= 1;
  c->cur ^= 1;
  return NEKGPU_OK;
}

}  // namespace nekgpu
