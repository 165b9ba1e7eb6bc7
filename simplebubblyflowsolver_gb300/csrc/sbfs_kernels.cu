// sm_103a kernels of the 2-D two-phase (VOF) time step.
//
// All arithmetic is FP64.  On GB300 the FP64 pipe (about 0.5 T fused
// multiply-adds per second, measured) bounds this solver, not HBM (a first
// version of the momentum kernel ran its FP64 pipe at 86% of peak with DRAM
// at 9%), so every kernel is written to spend as few FP64 instructions per
// cell as the discretisation allows, and on large launches half of the sums
// and products of the largest kernels run on the integer pipes beside it, bit
// for bit (sbfs_intfp.cuh):
//   * the reference's metric factors are folded into one coefficient per
//     column or per grid (see sbfs_device.cuh), and constant factors such
//     as the 0.5 of face averages are folded into those coefficients;
//   * reciprocals and inverse square roots are Newton-Raphson refinements of
//     the hardware seeds (rcp_nr, rsqrt_nr);
//   * 1 / rho^{k+1} is formed once per face and substage, and stored as
//     e = rho_ref / rho - 1, the factor the Poisson right-hand side and the
//     velocity correction both need;
//   * the THINC indicator 0.5 (1 + tanh(n . x + d)) with the intercept
//     d = -ln(1/phi - 1) / 2 equals 1 / (1 + K exp(-2 n . x)), K = 1/phi - 1:
//     one exponential per Gauss point and no logarithm;
//   * threshold tests (vofmin, upwind sign, clipping) run on the integer
//     pattern of the double; cells whose stencil inputs are bitwise equal
//     (single-phase bulk) take the exact short cut.
// The reference file:line each kernel follows is cited at the kernel.
#include <cooperative_groups.h>

#include <algorithm>
#include <cfloat>
#include <type_traits>

#include "sbfs_kernels.cuh"

namespace sbfs {

int g_pdl = 1;  // step kernels launched with programmatic stream serialisation
int g_stream_prio = 1;
int g_compact = -1;

namespace {

constexpr int BX = 32, BY = 8;

__device__ __forceinline__ size_t ix(const Grid &g, int row, int col) { return (size_t)row * g.p1 + col; }
__device__ __forceinline__ bool same(double a, double b) { return dbits(a) == dbits(b); }
// all of them zero, of either sign (by words)
template <class... T>
__device__ __forceinline__ bool zeros(T... x) {
  const unsigned hi = (... | intfp::high(intfp::bits(x))), lo = (... | intfp::low(intfp::bits(x)));
  return ((hi << 1) | lo) == 0u;
}

// Interface-branch compaction.  An FP64 instruction costs its warp an issue
// slot however few of its lanes run it (measured: eight FMA chains on 1 to
// 32 lanes of every warp all took the same time), and the cells that need
// the FP64 work of an interface branch lie along the interface and its THINC
// tails, often a few to a warp.  block_compact lists the block's threads
// whose flag is set in list[0 .. n) in thread order (a ballot per warp, a
// prefix over the warp counts in shared memory) and returns n, so that
// threads 0 .. n-1 can each take one listed cell and fill whole warps.
// Every thread of the block must call it (two barriers).
__device__ __forceinline__ int block_compact(bool flag, int tid, int *cnt, int *list) {
  const int lane = tid & 31, warp = tid >> 5, nwarp = (blockDim.x * blockDim.y + 31) >> 5;
  const unsigned mask = __ballot_sync(0xffffffffu, flag);
  if (lane == 0) cnt[warp] = __popc(mask);
  __syncthreads();
  int off = 0, n = 0;
  for (int w = 0; w < nwarp; ++w) {
    const int c = cnt[w];
    off += w < warp ? c : 0;
    n += c;
  }
  if (flag) list[off + __popc(mask & ((1u << lane) - 1u))] = tid;
  __syncthreads();
  return n;
}

dim3 grid2d(int ni, int nj, int nz = 1) { return dim3((ni + BX - 1) / BX, (nj + BY - 1) / BY, nz); }
// grid of the block shape of kernel k
dim3 tile_block(const Tiles &t, int k) { return dim3(t.bx[k], t.by[k]); }
dim3 tile_grid(const Tiles &t, int k, int ni, int nj, int nz) {
  return dim3((ni + t.bx[k] - 1) / t.bx[k], (nj + t.by[k] - 1) / t.by[k], nz);
}

// ---------------------------------------------------------------------------
// density, viscosity, corner gradients of vof
//   den:   src/fluid/density.c:9-31
//   visux: src/fluid/viscosity.c:23-61, visuy: :63-91
//   dvof:  src/interface/curvature_tensor.c:16-49
// thread (I, J): I = 0..nx+1
// ---------------------------------------------------------------------------
// unit normal of the vof gradient at the corner between columns I-1, I and
// rows J-1, J of a case (curvature_tensor.c:16-49)
__device__ __forceinline__ void corner_normal(const Grid &g, const Metrics &m, const double *__restrict__ vof,
                                              double *__restrict__ dvof, int zr, int I, int J) {
  const int r = J - 1 + zr, rm = wrap(J - 1, g.ny) + zr;
  const double a = vof[ix(g, rm, I - 1)], b = vof[ix(g, rm, I)];
  const double c = vof[ix(g, r, I - 1)], d = vof[ix(g, r, I)];
  // the reference's summation order, kept on purpose: in the THINC tails the
  // four values differ by ~1e-16 and the reference's sum is rounding noise
  // that the normalisation below (by max(|g|, eps)) scales up to O(1);
  // another order gives O(1) different corner normals
  const Fp64 f(I);
  const double gx = f.mul(m.ihxxf[I], f.add(f.sub(f.sub(b, a), c), d));
  const double gy = f.mul(f.reg(g.ihy), f.add(f.add(f.sub(-a, b), c), d));
  const double inv = inv_norm(fma(gx, gx, f.mul(gy, gy)), f);
  reinterpret_cast<double2 *>(dvof)[(size_t)r * (g.p2 / 2) + (I - 1)] = make_double2(f.mul(gx, inv), f.mul(gy, inv));
}

// compact: the corners with a gradient are handed to the block's first
// threads (see the interface-branch compaction below); otherwise each thread
// does its own.  The same arithmetic either way.  SCALED: the fused step's
// viscosities, visux times 2 nu / hy and visuy times 4 nu / hy (the factors
// k_momflux would otherwise apply per cell), formed with the constants and
// clip bounds scaled alike: the same two FP64 operations per face
template <bool DEN, bool VIS, bool GRAD, bool SCALED = false>
__global__ void __launch_bounds__(BX *BY) k_props(Grid g, Metrics m, Phys ph0, const double *__restrict__ vof,
                                                  double *__restrict__ den, double *__restrict__ visux,
                                                  double *__restrict__ visuy, double *__restrict__ dvof,
                                                  int compact, int *__restrict__ counts) {
  pdl_entry();
  // the interface cell and face counts k_curv_list adds to start at zero (a
  // memset between the two would end their programmatic dependency: 5 us on
  // the side stream of a 64 x 64 step)
  if (counts && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && threadIdx.y == 0) {
    counts[blockIdx.z] = 0;
    counts[g.nc + blockIdx.z] = 0;
  }
  const Phys ph = zphys(g, ph0);
  const int I = blockIdx.x * blockDim.x + threadIdx.x;
  const int J = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const bool in = I <= g.nx + 1 && J <= g.ny;
  const bool cmp = GRAD && compact;  // uniform over the block
  if (!cmp && !in) return;  // when compacting, every thread meets the barriers below
  const int zr = blockIdx.z * g.ny;  // first row of this case
  const int r = J - 1 + zr, rm = wrap(J - 1, g.ny) + zr;
  const Fp64 f(I);
  bool need = false;  // the corner gradient is not identically zero
  if (in) {
    const double v = vof[ix(g, r, I)];
    if (DEN) den[ix(g, r, I)] = clip_pos(fma(f.reg(ph.dm1), v, f.one), ph.den_lo, ph.den_hi);
    if (VIS) {
      // 1 + (visr - 1) 0.5 (a + b) = 1 + c2 (a + b), c2 = (visr - 1) / 2
      const double c = SCALED ? ph.vsx_c : ph.vm1, c2 = f.reg(SCALED ? ph.vsx_c2 : ph.hvm1);
      const double one = SCALED ? f.reg(ph.vsx_1) : f.one;
      if (I >= 1) {
        double vis;
        if (I == 1) vis = fma(c, vof[ix(g, r, 0)], one);
        else if (I == g.nx + 1) vis = fma(c, v, one);
        else vis = fma(c2, f.add(vof[ix(g, r, I - 1)], v), one);
        visux[ix(g, r, I - 1)] = SCALED ? clip_pos(vis, ph.vsx_lo, ph.vsx_hi) : clip_pos(vis, ph.vis_lo, ph.vis_hi);
      }
      const double vy = fma(SCALED ? f.reg(ph.vsy_c2) : c2, f.add(vof[ix(g, rm, I)], v), SCALED ? f.reg(ph.vsy_1) : f.one);
      visuy[ix(g, r, I)] = SCALED ? clip_pos(vy, ph.vsy_lo, ph.vsy_hi) : clip_pos(vy, ph.vis_lo, ph.vis_hi);
    }
    if (GRAD && I >= 1) {
      // zero where the four values are bitwise equal (single-phase bulk)
      const double a = vof[ix(g, rm, I - 1)], b = vof[ix(g, rm, I)], c = vof[ix(g, r, I - 1)];
      need = !(same(a, b) && same(b, c) && same(c, v));
      if (!need) reinterpret_cast<double2 *>(dvof)[(size_t)r * (g.p2 / 2) + (I - 1)] = make_double2(0., 0.);
      else if (!cmp) corner_normal(g, m, vof, dvof, zr, I, J);
    }
  }
  if (cmp) {
    __shared__ int cnt[BX * BY / 32];
    __shared__ int list[BX * BY];
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    const int n = block_compact(need, tid, cnt, list);
    if (tid < n) {
      const int sy = list[tid] / blockDim.x, sx = list[tid] - sy * blockDim.x;
      corner_normal(g, m, vof, dvof, zr, blockIdx.x * blockDim.x + sx, blockIdx.y * blockDim.y + sy + 1);
    }
  }
}

// ---------------------------------------------------------------------------
// cell normal + THINC parameter (interface cells) and curvature
//   normal:    src/interface/curvature_tensor.c:51-97
//   curvature: src/interface/curvature_tensor.c:100-135
//     kappa = -[(nx_xp - nx_xm) / HXXC + (ny_yp - ny_ym) / hy]
// STORE_K: the third component is K = 1/phi - 1 (used by the fused step);
// otherwise the reference's intercept d = -ln(1/phi - 1) / 2.
// thread (I, J): I = 1..nx
// ---------------------------------------------------------------------------
template <bool NORMAL, bool CURV, bool STORE_K>
__global__ void __launch_bounds__(BX *BY) k_normal_curv(Grid g, Metrics m, const double *__restrict__ vof,
                                                        const double *__restrict__ dvof, double *__restrict__ normal,
                                                        double *__restrict__ curv) {
  pdl_entry();
  const int I = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int J = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (I > g.nx || J > g.ny) return;
  const int r = J - 1, rp = wrap(J + 1, g.ny);
  const double2 *dv = reinterpret_cast<const double2 *>(dvof);
  const size_t q = g.p2 / 2;
  const double2 d00 = dv[(size_t)r * q + (I - 1)], d10 = dv[(size_t)r * q + I];
  const double2 d01 = dv[(size_t)rp * q + (I - 1)], d11 = dv[(size_t)rp * q + I];
  if (CURV) {
    const long long any = dbits(d00.x) | dbits(d00.y) | dbits(d10.x) | dbits(d10.y) | dbits(d01.x) | dbits(d01.y) |
                          dbits(d11.x) | dbits(d11.y);
    double k = -0.;
    if ((any << 1) != 0) {  // some corner normal is not +-0
      const double ddx = (d10.x + d11.x) - (d00.x + d01.x);
      const double ddy = (d01.y + d11.y) - (d00.y + d10.y);
      k = -fma(m.hihxxc[I], ddx, g.hihy * ddy);
    }
    curv[ix(g, r, I)] = k;
  }
  if (NORMAL) {
    const double phi = vof[ix(g, r, I)];
    if (!single_phase(phi)) {
      const double mx = (((d00.x + d10.x) + d01.x) + d11.x) * m.ihxxc[I];
      const double my = (((d00.y + d10.y) + d01.y) + d11.y) * g.ihy;
      const double inv = inv_norm(fma(mx, mx, my * my));
      double *o = normal + (size_t)r * g.p3 + (size_t)(I - 1) * 3;
      o[0] = mx * inv;
      o[1] = my * inv;
      o[2] = STORE_K ? rcp_nr(phi) - 1. : -0.5 * log(__drcp_rn(phi) - 1.);
    }
  }
}

// THINC flux factor of one face (src/interface/update/main.c:18-35,
// fluxx.c:62-68): the mean of the indicator over the two Gauss points
// t = +-g of the face, 0.5 sum 1 / (1 + K exp(-2 (n_a s + n_b t))), where s
// is the face position along its normal (+-1/2) and n_a, n_b the normal
// components along and across it.  With a = K exp(-2 n_a s) and
// b = exp(-2 n_b g) the two terms are 1 / (1 + a b) and b / (b + a).
// The caller passes -2 n_a s, which for s = -+1/2 is exactly +-n_a.
__device__ __forceinline__ double thinc_ab(double a, double b) {
  const double p = fma(a, b, 1.);
  const double q = b + a;
  // b p + q >= b >= exp(-2 g) > 1/2: positive and normal
  return half_pos_normal(fma(b, p, q)) * rcp_nr(p * q);
}
// a is rounded on its own (never fused into q = b + a), so that a factor
// formed ahead of time (k_curv_list<false>) gives the same flux
__device__ __forceinline__ double thinc_face(double m2nas, double nb, double K) {
  return thinc_ab(__dmul_rn(K, exp(m2nas)), exp(-2. * kGaussPt * nb));
}

// ---------------------------------------------------------------------------
// THINC vof fluxes and CSF surface-tension force
//   fluxes: src/interface/update/fluxx.c:14-73, fluxy.c:14-73
//   force:  src/interface/force.c:20-88
// HAVE_K: normal[2] holds K = 1/phi - 1 (fused step) instead of the
// reference's intercept d (then K = exp(-2 d)).
// thread (I, J): I = 1..nx handles x face I (I >= 2) and y face (I, J - 1/2)
// ---------------------------------------------------------------------------
// ITF_KAPPA (learned curvature mode): the face curvature comes from the
// interface side alone when only one of the two cells is an interface cell
// (the -div n of a single-phase cell next to the interface is not a
// curvature of anything); otherwise the mean, as in the reference.
__device__ __forceinline__ double face_kappa_sum(double pl, double pr, double kl, double kr) {
  const bool il = !single_phase(pl), ir = !single_phase(pr);
  return il == ir ? kl + kr : (il ? 2. * kl : 2. * kr);
}

template <bool FLUX, bool FORCE, bool HAVE_K, bool BULK_ONLY, bool ITF_KAPPA>
__device__ __forceinline__ void flux_force_body(const Grid &g, const Metrics &m, const Phys &ph0,
                                                const double *__restrict__ ux, const double *__restrict__ uy,
                                                const double *__restrict__ vof, const double *__restrict__ normal,
                                                const double *__restrict__ den0, const double *__restrict__ curv,
                                                double *__restrict__ fluxx, double *__restrict__ fluxy,
                                                double *__restrict__ ifrcx, double *__restrict__ ifrcy) {
  const Phys ph = zphys(g, ph0);
  const int I = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int J = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (I > g.nx || J > g.ny) return;
  const int zr = blockIdx.z * g.ny;  // first row of this case
  const int r = J - 1 + zr, rm = wrap(J - 1, g.ny) + zr;
  const double v0 = vof[ix(g, r, I)];
  const double vxm = vof[ix(g, r, I - 1)];
  const double vym = vof[ix(g, rm, I)];
  if (FLUX) {
    if (I >= 2) {
      const double vel = ux[ix(g, r, I - 1)];
      const bool n = neg(vel);
      const int iu = n ? I : I - 1;
      const double phi = n ? v0 : vxm;
      if (single_phase(phi)) {
        fluxx[ix(g, r, I - 1)] = vel * phi;
      } else if (!BULK_ONLY) {
        const double *nv = normal + (size_t)r * g.p3 + (size_t)(iu - 1) * 3;
        const double K = HAVE_K ? nv[2] : exp(-2. * nv[2]);
        fluxx[ix(g, r, I - 1)] = vel * thinc_face(n ? nv[0] : -nv[0], nv[1], K);
      }
    }
    {
      const double vel = uy[ix(g, r, I)];
      const bool n = neg(vel);
      const int ru = n ? r : rm;
      const double phi = n ? v0 : vym;
      if (single_phase(phi)) {
        fluxy[ix(g, r, I)] = vel * phi;
      } else if (!BULK_ONLY) {
        const double *nv = normal + (size_t)ru * g.p3 + (size_t)(I - 1) * 3;
        const double K = HAVE_K ? nv[2] : exp(-2. * nv[2]);
        fluxy[ix(g, r, I)] = vel * thinc_face(n ? nv[1] : -nv[1], nv[0], K);
      }
    }
    // impermeable walls / dummy ghost faces
    if (I == 1) {
      fluxx[ix(g, r, 0)] = 0.;
      fluxy[ix(g, r, 0)] = 0.;
    }
    if (I == g.nx) {
      fluxx[ix(g, r, g.nx)] = 0.;
      fluxy[ix(g, r, g.nx + 1)] = 0.;
    }
  }
  if (FORCE) {
    const Fp64 w(I);
    // f = 0.5 (rho_l + rho_r) 2 / (1 + denr) / We 0.5 (k_l + k_r) (phi_r - phi_l) / h
    if (I >= 2) {
      double f = 0.;
      if (!same(vxm, v0)) {
        const double rho = w.add(den0[ix(g, r, I - 1)], den0[ix(g, r, I)]);
        const double kap = ITF_KAPPA ? face_kappa_sum(vxm, v0, curv[ix(g, r, I - 1)], curv[ix(g, r, I)])
                                     : w.add(curv[ix(g, r, I - 1)], curv[ix(g, r, I)]);
        f = w.mul(w.mul(rho, kap), w.mul(w.mul(w.reg(ph.qf), m.ihxxf[I]), w.sub(v0, vxm)));
      }
      ifrcx[ix(g, r, I - 2)] = f;
    }
    double f = 0.;
    if (!same(vym, v0)) {
      const double rho = w.add(den0[ix(g, rm, I)], den0[ix(g, r, I)]);
      const double kap = ITF_KAPPA ? face_kappa_sum(vym, v0, curv[ix(g, rm, I)], curv[ix(g, r, I)])
                                   : w.add(curv[ix(g, rm, I)], curv[ix(g, r, I)]);
      f = w.mul(w.mul(rho, kap), w.mul(w.reg(ph.qfy), w.sub(v0, vym)));
    }
    ifrcy[ix(g, r, I - 1)] = f;
  }
}

template <bool FLUX, bool FORCE, bool HAVE_K, bool BULK_ONLY = false, bool ITF_KAPPA = false>
__global__ void __launch_bounds__(BX *BY)
    k_flux_force(Grid g, Metrics m, Phys ph0, const double *__restrict__ ux, const double *__restrict__ uy,
                 const double *__restrict__ vof, const double *__restrict__ normal, const double *__restrict__ den0,
                 const double *__restrict__ curv, double *__restrict__ fluxx, double *__restrict__ fluxy,
                 double *__restrict__ ifrcx, double *__restrict__ ifrcy) {
  pdl_entry();
  flux_force_body<FLUX, FORCE, HAVE_K, BULK_ONLY, ITF_KAPPA>(g, m, ph0, ux, uy, vof, normal, den0, curv, fluxx, fluxy,
                                                             ifrcx, ifrcy);
}

// the fluxes of the faces whose upwind cell is single-phase (flux = vel phi)
// and the wall faces; the faces of upwind interface cells are k_face_flux's
__global__ void __launch_bounds__(BX *BY)
    k_bulk_flux(Grid g, Metrics m, Phys ph0, const double *__restrict__ ux, const double *__restrict__ uy,
                const double *__restrict__ vof, double *__restrict__ fluxx, double *__restrict__ fluxy) {
  pdl_entry();
  flux_force_body<true, false, true, true, false>(g, m, ph0, ux, uy, vof, nullptr, nullptr, nullptr, fluxx, fluxy,
                                                  nullptr, nullptr);
}

// the CSF force alone (it needs no velocity), into the force buffers given
template <bool ITF_KAPPA>
__global__ void __launch_bounds__(BX *BY)
    k_csf_force(Grid g, Metrics m, Phys ph0, const double *__restrict__ vof, const double *__restrict__ den0,
                const double *__restrict__ curv, double *__restrict__ ifrcx, double *__restrict__ ifrcy) {
  pdl_entry();
  flux_force_body<false, true, false, false, ITF_KAPPA>(g, m, ph0, nullptr, nullptr, vof, nullptr, den0, curv,
                                                        nullptr, nullptr, ifrcx, ifrcy);
}

// ---------------------------------------------------------------------------
// Interface compaction of the fused step.  THINC work (normal, intercept,
// two exponentials per face) exists only in interface cells, a few percent
// of the domain scattered along the bubbles; done in place it makes whole
// warps wait on a few lanes.  Two arrangements, the same arithmetic:
// listed faces (the step's first form):
//   k_curv_list<true> curvature of every cell (curvature_tensor.c:100-135),
//                     a list of the interface cells and a list of the faces
//                     they are upwind of (block-aggregated appends)
//   k_interface_cells one thread per listed face: the cell's normal and
//                     K = 1/phi - 1 (curvature_tensor.c:51-97), then the THINC
//                     flux of that face (update/fluxx.c, fluxy.c); a cell
//                     with two upwind faces is set up twice, but no warp
//                     runs a face branch only some of its lanes take
//   k_flux_force<.., BULK_ONLY>  every other face (upwind cell single-phase:
//                     flux = vel phi) and the CSF force
// Each face is written by exactly one of them: the upwind choice and the
// vofmin test are the same integer tests in both.
// geometry ahead (the default): everything but the upwind choice depends on
// vof alone, so it runs beside the previous substage's predictor and
// Poisson solve, and no flux kernel stands between the correction and the
// VOF update:
//   k_curv_list<false> curvature, the interface-cell list and per interface
//                     cell its THINC factors K exp(+-n_a) for its four faces
//                     and exp(-2 g n_b) across x and y faces (the block's
//                     interface cells handed to its first threads)
//   k_csf_force       the CSF force
//   k_face_flux       one thread per face of a listed cell: the upwind test,
//                     then the THINC flux from the cell's factors
//   k_bulk_flux       every other face, as k_flux_force<.., BULK_ONLY>
// ---------------------------------------------------------------------------
// kappa = -div n of cell (I, J) of a case from its four corner normals
// (curvature_tensor.c:100-135)
__device__ __forceinline__ void cell_curv(const Grid &g, const Metrics &m, const double2 *__restrict__ dv,
                                          double *__restrict__ curv, int zr, int I, int J) {
  const size_t q = g.p2 / 2;
  const int r = J - 1 + zr, rp = wrap(J + 1, g.ny) + zr;
  const double2 d00 = dv[(size_t)r * q + (I - 1)], d10 = dv[(size_t)r * q + I];
  const double2 d01 = dv[(size_t)rp * q + (I - 1)], d11 = dv[(size_t)rp * q + I];
  const Fp64 f(I);
  const double ddx = f.sub(f.add(d10.x, d11.x), f.add(d00.x, d01.x));
  const double ddy = f.sub(f.add(d01.y, d11.y), f.add(d00.y, d10.y));
  curv[ix(g, r, I)] = -fma(m.hihxxc[I], ddx, f.mul(f.reg(g.hihy), ddy));
}

// unit normal (n0, n1) and K = 1/phi - 1 of interface cell (I, J) of a case
// (curvature_tensor.c:51-97)
__device__ __forceinline__ void cell_normal_k(const Grid &g, const Metrics &m, const double2 *__restrict__ dv,
                                              const double *__restrict__ vof, int zr, int I, int J, double &n0,
                                              double &n1, double &K) {
  const size_t q = g.p2 / 2;
  const int r = J - 1 + zr, rp = wrap(J + 1, g.ny) + zr;
  const double2 d00 = dv[(size_t)r * q + (I - 1)], d10 = dv[(size_t)r * q + I];
  const double2 d01 = dv[(size_t)rp * q + (I - 1)], d11 = dv[(size_t)rp * q + I];
  const double mx = (((d00.x + d10.x) + d01.x) + d11.x) * m.ihxxc[I];
  const double my = (((d00.y + d10.y) + d01.y) + d11.y) * g.ihy;
  const double inv = inv_norm(fma(mx, mx, my * my));
  n0 = mx * inv;
  n1 = my * inv;
  K = rcp_nr(vof[ix(g, r, I)]) - 1.;
}

// THINC factors of interface cell (I, J), stored at its cell index `at`
// (planar, cap entries a table, kThincTabs of them): a of its left, right,
// bottom and top faces (thinc_face's K exp(-2 n_a s)), then b of its x and
// of its y faces
__device__ __forceinline__ void cell_thinc_factors(const Grid &g, const Metrics &m, const double2 *__restrict__ dv,
                                                   const double *__restrict__ vof, int zr, int I, int J,
                                                   double *__restrict__ tf, size_t cap, int at) {
  double n0, n1, K;
  cell_normal_k(g, m, dv, vof, zr, I, J, n0, n1, K);
  tf[at] = __dmul_rn(K, exp(n0));
  tf[cap + at] = __dmul_rn(K, exp(-n0));
  tf[2 * cap + at] = __dmul_rn(K, exp(n1));
  tf[3 * cap + at] = __dmul_rn(K, exp(-n1));
  tf[4 * cap + at] = exp(-2. * kGaussPt * n1);
  tf[5 * cap + at] = exp(-2. * kGaussPt * n0);
}

// compact: the cells with a corner normal hand their curvature to the
// block's first threads (interface-branch compaction); otherwise each thread
// computes its own.  The same arithmetic either way.
// FACES: also the list of the faces the interface cells are upwind of (from
// the velocity); else, without the velocity, the THINC factors of every
// interface cell (tables by cell index), by the block's first threads
template <bool FACES>
__global__ void __launch_bounds__(BX *BY) k_curv_list(Grid g, Metrics m, const double *__restrict__ vof,
                                                      const double *__restrict__ dvof, const double *__restrict__ ux,
                                                      const double *__restrict__ uy, double *__restrict__ curv,
                                                      int *__restrict__ list, int *__restrict__ count,
                                                      int *__restrict__ flist, int *__restrict__ fcount,
                                                      double *__restrict__ tf, int compact) {
  pdl_entry();
  const size_t cap = (size_t)g.nx * g.ny;
  list += (size_t)blockIdx.z * cap;
  count += (size_t)blockIdx.z * (1);
  if (FACES) {
    flist += (size_t)blockIdx.z * (4 * cap);
    fcount += (size_t)blockIdx.z * (1);
  } else {
    tf += (size_t)blockIdx.z * (kThincTabs * cap);
  }
  const int I = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int J = blockIdx.y * blockDim.y + threadIdx.y + 1;
  const bool in = I <= g.nx && J <= g.ny;
  const int zr = blockIdx.z * g.ny;
  const double2 *dv = reinterpret_cast<const double2 *>(dvof);
  const size_t q = g.p2 / 2;
  bool itf = false, kap = false;  // kap: some corner normal of the cell is not +-0
  unsigned up = 0u;  // faces this cell is upwind of: bit 0 left, 1 right, 2 bottom, 3 top
  if (in) {
    const int r = J - 1 + zr, rp = wrap(J + 1, g.ny) + zr;
    const double2 d00 = dv[(size_t)r * q + (I - 1)], d10 = dv[(size_t)r * q + I];
    const double2 d01 = dv[(size_t)rp * q + (I - 1)], d11 = dv[(size_t)rp * q + I];
    const long long any = dbits(d00.x) | dbits(d00.y) | dbits(d10.x) | dbits(d10.y) | dbits(d01.x) | dbits(d01.y) |
                          dbits(d11.x) | dbits(d11.y);
    kap = (any << 1) != 0;
    if (!kap) curv[ix(g, r, I)] = -0.;
    else if (!compact) cell_curv(g, m, dv, curv, zr, I, J);
    itf = !single_phase(vof[ix(g, r, I)]);
    if (FACES && itf) {
      // upwind tests of update/fluxx.c, fluxy.c; the wall faces belong to k_flux_force
      up |= (I >= 2 && neg(ux[ix(g, r, I - 1)])) ? 1u : 0u;
      up |= (I < g.nx && !neg(ux[ix(g, r, I)])) ? 2u : 0u;
      up |= neg(uy[ix(g, r, I)]) ? 4u : 0u;
      up |= !neg(uy[ix(g, rp, I)]) ? 8u : 0u;
    }
  }
  // block-aggregated appends: per warp (32 consecutive threads of the block,
  // whatever its shape) the ballots of its cells and faces, per block one
  // atomic per list; the order of the entries is free (each is processed on
  // its own)
  const int tid = threadIdx.y * blockDim.x + threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5, nwarp = (blockDim.x * blockDim.y + 31) >> 5;
  const int cell = (J - 1) * g.nx + (I - 1);
  const unsigned below = (1u << lane) - 1u;
  const unsigned kmask = __ballot_sync(0xffffffffu, kap);
  const unsigned mask = __ballot_sync(0xffffffffu, itf);
  unsigned fm[4] = {0u, 0u, 0u, 0u};
  int nfw = 0;
  if (FACES) {
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      fm[f] = __ballot_sync(0xffffffffu, (up >> f) & 1u);
      nfw += __popc(fm[f]);
    }
  }
  // per warp: its interface cell / face / curvature cell count, then its
  // offset in the block (lists) or among the block's curvature cells
  __shared__ int wofs[3][BX * BY / 32];
  __shared__ int bbase[3], btot[3];
  __shared__ int klist[BX * BY];
  __shared__ int ilocal[FACES ? 1 : BX * BY];
  if (lane == 0) {
    wofs[0][warp] = __popc(mask);
    wofs[1][warp] = nfw;
    wofs[2][warp] = __popc(kmask);
  }
  __syncthreads();
  if (tid < 3) {
    int run = 0;
    for (int w = 0; w < nwarp; ++w) {
      const int c = wofs[tid][w];
      wofs[tid][w] = run;
      run += c;
    }
    btot[tid] = run;
    bbase[tid] = tid == 2 ? run : (run ? atomicAdd(tid == 0 ? count : fcount, run) : 0);
  }
  __syncthreads();
  const int ipos = wofs[0][warp] + __popc(mask & below);  // this cell's place among the block's interface cells
  if (itf) list[bbase[0] + ipos] = cell;
  if (FACES) {
    int fo = bbase[1] + wofs[1][warp];
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      if ((up >> f) & 1u) flist[fo + __popc(fm[f] & below)] = 4 * cell + f;
      fo += __popc(fm[f]);
    }
  } else if (itf) {
    ilocal[ipos] = tid;
  }
  // compacted curvature: the cells with a corner normal lie in the THINC
  // tails, often a few to a warp (the prefix of their counts came with the
  // lists' above)
  if (compact && kap) klist[wofs[2][warp] + __popc(kmask & below)] = tid;
  if (!FACES || compact) __syncthreads();  // uniform over the block
  if (compact && tid < bbase[2]) {
    const int sy = klist[tid] / blockDim.x, sx = klist[tid] - sy * blockDim.x;
    cell_curv(g, m, dv, curv, zr, blockIdx.x * blockDim.x + sx + 1, blockIdx.y * blockDim.y + sy + 1);
  }
  // the THINC factors of the block's interface cells
  if (!FACES && tid < btot[0]) {
    const int c = ilocal[tid];
    const int sy = c / blockDim.x, sx = c - sy * blockDim.x;
    const int Ic = blockIdx.x * blockDim.x + sx + 1, Jc = blockIdx.y * blockDim.y + sy + 1;
    cell_thinc_factors(g, m, dv, vof, zr, Ic, Jc, tf, cap, (Jc - 1) * g.nx + (Ic - 1));
  }
}

__global__ void __launch_bounds__(256)
    k_interface_cells(Grid g, Metrics m, const double *__restrict__ ux, const double *__restrict__ uy,
                      const double *__restrict__ vof, const double *__restrict__ dvof, const int *__restrict__ flist,
                      const int *__restrict__ fcount, double *__restrict__ fluxx, double *__restrict__ fluxy) {
  pdl_entry();
  flist += (size_t)blockIdx.z * (4 * (size_t)g.nx * g.ny);
  fcount += (size_t)blockIdx.z * (1);
  const int n = *fcount;
  const int zr = blockIdx.z * g.ny;  // first row of this case
  const double2 *dv = reinterpret_cast<const double2 *>(dvof);
  // one thread per upwind face of an interface cell: every thread runs the
  // same instructions (no face branches)
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    const int code = flist[t];
    const int id = code >> 2, f = code & 3;
    const int r0 = id / g.nx, I = id - r0 * g.nx + 1;
    const int J = r0 + 1, r = r0 + zr, rp = wrap(J + 1, g.ny) + zr;
    double n0, n1, K;
    cell_normal_k(g, m, dv, vof, zr, I, J, n0, n1, K);
    // face f: 0 left (x face I), 1 right (x face I + 1), 2 bottom (y face J - 1/2), 3 top (J + 1/2)
    const bool xf = f < 2;
    const double na = xf ? n0 : n1, nb = xf ? n1 : n0;
    const double ena = (f & 1) ? -na : na;  // -2 n_a s with s = -1/2 (left, bottom) or +1/2
    const size_t at = xf ? ix(g, r, I - 1 + f) : ix(g, f == 2 ? r : rp, I);
    const double vel = xf ? ux[at] : uy[at];
    const double fl = vel * thinc_face(ena, nb, K);
    if (xf)
      fluxx[at] = fl;
    else
      fluxy[at] = fl;
  }
}

// ---------------------------------------------------------------------------
// vof source (flux divergence), RK update and vof boundaries
//   src/interface/update/main.c:54-136, src/interface/boundary.c:15-42
//   src = (F_x(i) - F_x(i+1)) / HXXC + (F_y(j) - F_y(j+1)) / hy
// FUSED additionally writes rho^{k+1} (src/fluid/density.c) and the mass
// fluxes u + (rho_r - 1) flux into separate buffers
// (src/interface/mass_flux.c:10-58).  OUT: vof^{k+1} goes to vof_out
// (the geometry-ahead step, whose side stream still reads vof^k), else in
// place.
// thread (I, J): I = 1..nx
// ---------------------------------------------------------------------------
template <bool FUSED, bool OUT, bool INT>
__global__ void __launch_bounds__(BX *BY)
    k_vof_advance(Grid g, Metrics m, Phys ph0, const double *__restrict__ sc, int k, double *vof, double *vof_out,
                  const double *__restrict__ fluxx, const double *__restrict__ fluxy, double *__restrict__ src_a,
                  const double *__restrict__ src_b, const double *__restrict__ ux, const double *__restrict__ uy,
                  double *__restrict__ mfx, double *__restrict__ mfy, double *__restrict__ den1) {
  pdl_entry();
  const Phys ph = zphys(g, ph0);
  sc += (size_t)blockIdx.z * (kScalars);
  const int I = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int J = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (I > g.nx || J > g.ny) return;
  const int zr = blockIdx.z * g.ny;  // first row of this case
  const int r = J - 1 + zr, rp = wrap(J + 1, g.ny) + zr;
  const double fxm = fluxx[ix(g, r, I - 1)], fxp = fluxx[ix(g, r, I)];
  const double fym = fluxy[ix(g, r, I)], fyp = fluxy[ix(g, rp, I)];
  const Fp64 f(I);
  Fp64Int<INT> q(f);
  const double ihy = f.reg(g.ihy), dfy = f.sub(fym, fyp);
  // two of the nine FP64 operations on the integer pipes (2048 x 1024, one
  // launch, 40.3 -> 33.6 us; a third 35.1 us)
  double dx = q.subz(fxm, fxp), dy = q.mulz(ihy, dfy);
  if (INT && q.bad) {
    dx = rare_add(fxm, -fxp);
    dy = rare_mul(ihy, dfy);
  }
  const double s = fma(m.ihxxc[I], dx, dy);
  src_a[ix(g, r, I - 1)] = s;
  double v = vof[ix(g, r, I)];
  v = fma(sc[sc_adt(k)], s, v);
  if (k != 0) v = fma(sc[sc_bdt(k)], src_b[ix(g, r, I - 1)], v);
  double *vo = OUT ? vof_out : vof;
  vo[ix(g, r, I)] = v;
  if (I == 1) vo[ix(g, r, 0)] = 0.;
  if (I == g.nx) vo[ix(g, r, g.nx + 1)] = 0.;
  if (FUSED) {
    const double c = f.reg(ph.dm1);
    den1[ix(g, r, I)] = clip_pos(fma(c, v, f.one), ph.den_lo, ph.den_hi);
    mfx[ix(g, r, I - 1)] = fma(c, fxm, ux[ix(g, r, I - 1)]);
    mfy[ix(g, r, I)] = fma(c, fym, uy[ix(g, r, I)]);
    if (I == 1) {
      den1[ix(g, r, 0)] = clip_pos(1., ph.den_lo, ph.den_hi);
      mfy[ix(g, r, 0)] = fma(c, fluxy[ix(g, r, 0)], uy[ix(g, r, 0)]);
    }
    if (I == g.nx) {
      den1[ix(g, r, g.nx + 1)] = clip_pos(1., ph.den_lo, ph.den_hi);
      mfx[ix(g, r, g.nx)] = fma(c, fxp, ux[ix(g, r, g.nx)]);
      mfy[ix(g, r, g.nx + 1)] = fma(c, fluxy[ix(g, r, g.nx + 1)], uy[ix(g, r, g.nx + 1)]);
    }
  }
}

// one thread per face of a listed interface cell (four per cell, face f = 0
// left, 1 right, 2 bottom, 3 top): the upwind test of update/fluxx.c and
// fluxy.c, then, where the cell is upwind of the face, its THINC flux from
// the cell's factors (k_curv_list<false>, tables by cell index) into fluxx /
// fluxy.  The wall faces carry no flux.  Each block takes a contiguous share
// of the entries, so that every SM gets some.
__global__ void __launch_bounds__(256)
    k_face_flux(Grid g, const double *__restrict__ ux, const double *__restrict__ uy, const int *__restrict__ list,
                const int *__restrict__ count, const double *__restrict__ tf, double *__restrict__ fluxx,
                double *__restrict__ fluxy) {
  pdl_entry();
  const size_t cap = (size_t)g.nx * g.ny;
  list += (size_t)blockIdx.z * cap;
  count += (size_t)blockIdx.z * (1);
  tf += (size_t)blockIdx.z * (kThincTabs * cap);
  const int n4 = 4 * *count;
  const int zr = blockIdx.z * g.ny;  // first row of this case
  const int per = ((n4 + (int)gridDim.x - 1) / (int)gridDim.x + 31) & ~31;
  const int t0 = blockIdx.x * per, t1 = min(n4, t0 + per);
  for (int t = t0 + threadIdx.x; t < t1; t += blockDim.x) {
    const int f = t & 3;
    const int id = list[t >> 2];
    const int r0 = id / g.nx, I = id - r0 * g.nx + 1;
    const int J = r0 + 1, r = r0 + zr, rp = wrap(J + 1, g.ny) + zr;
    const bool xf = f < 2;
    const size_t at = xf ? ix(g, r, I - 1 + f) : ix(g, f == 2 ? r : rp, I);
    const double vel = xf ? ux[at] : uy[at];
    const bool up = f == 0 ? (I >= 2 && neg(vel)) : (f == 1 ? (I < g.nx && !neg(vel)) : (f == 2 ? neg(vel) : !neg(vel)));
    if (!up) continue;
    const double fl = vel * thinc_ab(tf[f * cap + id], tf[(4 + (f >> 1)) * cap + id]);
    if (xf)
      fluxx[at] = fl;
    else
      fluxy[at] = fl;
  }
}

// vof flux -> mass flux in place (src/interface/mass_flux.c:10-58); I = 0..nx+1
__global__ void k_mass_flux(Grid g, Phys ph, const double *__restrict__ ux, const double *__restrict__ uy,
                            double *__restrict__ fluxx, double *__restrict__ fluxy) {
  pdl_entry();
  const int I = blockIdx.x * blockDim.x + threadIdx.x;
  const int J = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (I > g.nx + 1 || J > g.ny) return;
  const int r = J - 1;
  const double c = ph.denr - 1.;
  if (I >= 1) fluxx[ix(g, r, I - 1)] = fma(c, fluxx[ix(g, r, I - 1)], ux[ix(g, r, I - 1)]);
  fluxy[ix(g, r, I)] = fma(c, fluxy[ix(g, r, I)], uy[ix(g, r, I)]);
}

// ---------------------------------------------------------------------------
// viscous stress tensor: txx, tyy at centres, txy at corners
//   src/fluid/predict/txx.c:11-40, txy.c:13-50, tyy.c:10-38
//   txx = 2 mu du/dx = (mu_l + mu_r) (u_r - u_l) / HXXC, likewise tyy;
//   txy = 0.5 (mu_s + mu_n) du/dy + 0.5 (mu_w + mu_e) dv/dx
// thread (I, J): I = 1..nx+1
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(BX *BY)
    k_stress(Grid g, Metrics m, const double *__restrict__ ux, const double *__restrict__ uy,
             const double *__restrict__ visux, const double *__restrict__ visuy, double *__restrict__ txx,
             double *__restrict__ txy, double *__restrict__ tyy) {
  pdl_entry();
  const int I = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int J = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (I > g.nx + 1 || J > g.ny) return;
  const int zr = blockIdx.z * g.ny;  // first row of this case
  const int r = J - 1 + zr, rm = wrap(J - 1, g.ny) + zr, rp = wrap(J + 1, g.ny) + zr;
  const double u0 = ux[ix(g, r, I - 1)];
  const double vx0 = visux[ix(g, r, I - 1)];
  const double w0 = uy[ix(g, r, I)];
  const double vy0 = visuy[ix(g, r, I)];
  if (I <= g.nx) {
    txx[ix(g, r, I - 1)] = (vx0 + visux[ix(g, r, I)]) * ((ux[ix(g, r, I)] - u0) * m.ihxxc[I]);
    tyy[ix(g, r, I - 1)] = (vy0 + visuy[ix(g, rp, I)]) * ((uy[ix(g, rp, I)] - w0) * g.ihy);
  }
  const double sx = visux[ix(g, rm, I - 1)] + vx0;
  const double sy = visuy[ix(g, r, I - 1)] + vy0;
  const double lxy = (u0 - ux[ix(g, rm, I - 1)]) * g.hihy;
  const double lyx = (w0 - uy[ix(g, r, I - 1)]) * m.hihxxf[I];
  txy[ix(g, r, I - 1)] = fma(sx, lxy, sy * lyx);
}

// ---------------------------------------------------------------------------
// momentum right-hand sides and the RK predictor
//   ux: src/fluid/predict/ux.c:29-273, uy: src/fluid/predict/uy.c:29-251,
//   src/fluid/predict/main.c:9-80, walls: src/fluid/boundary/ux.c, uy.c
// With JD = H hy the ux terms reduce to
//   adv_x = 0.25 / HXXF(i) [(F_i + F_i+1)(u_i + u_i+1) - (F_i-1 + F_i)(u_i-1 + u_i)]
//   adv_y = 0.25 HXXC / (HXXF(i) hy) [(G_j+1 sums)(u_j + u_j+1) - (G_j sums)(u_j-1 + u_j)]
//   dif_x = nu / HXXF(i) (txx_i - txx_i-1),  dif_y = nu / hy (txy_j+1 - txy_j)
// and the uy terms likewise with HXXC in place of HXXF.
// This is the fine-grained entry point's form (fluid_predict_field returns
// txx, txy, tyy and the sources); the fused step uses k_momflux and
// k_predict_mf below, the same terms with every flux formed once.
// thread (I, J): I = 1..nx handles the ux face I (I >= 2) and the uy face
// (I, J - 1/2)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(BX *BY)
    k_predict(Grid g, Metrics m, Phys ph0, const double *__restrict__ sc, int k, const double *__restrict__ ux,
              const double *__restrict__ uy, double *__restrict__ ux_out, double *__restrict__ uy_out,
              const double *__restrict__ mfx, const double *__restrict__ mfy, const double *__restrict__ txx,
              const double *__restrict__ txy, const double *__restrict__ tyy, const double *__restrict__ p,
              const double *__restrict__ ifrcx, const double *__restrict__ ifrcy, const double *__restrict__ den0,
              const double *__restrict__ den1, double *__restrict__ sxa, const double *__restrict__ sxb,
              double *__restrict__ sxg, double *__restrict__ sya, const double *__restrict__ syb,
              double *__restrict__ syg) {
  pdl_entry();
  const Phys ph = zphys(g, ph0);
  const double *__restrict__ nuf = m.nuf + (size_t)blockIdx.z * g.cm;
  const double *__restrict__ nuc = m.nuc + (size_t)blockIdx.z * g.cm;
  sc += (size_t)blockIdx.z * (kScalars);
  const int I = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int J = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (I > g.nx || J > g.ny) return;
  const int zr = blockIdx.z * g.ny;  // first row of this case
  const int r = J - 1 + zr, rm = wrap(J - 1, g.ny) + zr, rp = wrap(J + 1, g.ny) + zr;
  // the update is carried as 2u with 2 alpha dt, ... and 1 / (2 rho_face):
  // powers of two, so every rounding is the one of the plain form
  const double adt2 = sc[sc_adt2(k)], bdt2 = sc[sc_bdt2(k)], gdt2 = sc[sc_gdt2(k)];
  const double nuy = ph.nuy;
  // ---- ux at face I
  if (I >= 2) {
    const double fx0 = mfx[ix(g, r, I - 1)];
    const double u0 = ux[ix(g, r, I - 1)];
    const double sxm = mfx[ix(g, r, I - 2)] + fx0, sxp = fx0 + mfx[ix(g, r, I)];
    const double um = ux[ix(g, r, I - 2)] + u0, up = u0 + ux[ix(g, r, I)];
    const double sym = mfy[ix(g, r, I - 1)] + mfy[ix(g, r, I)];
    const double syp = mfy[ix(g, rp, I - 1)] + mfy[ix(g, rp, I)];
    const double vm = ux[ix(g, rm, I - 1)] + u0, vp = u0 + ux[ix(g, rp, I - 1)];
    double a = ifrcx[ix(g, r, I - 2)];
    const double rho0 = den0[ix(g, r, I - 1)] + den0[ix(g, r, I)];  // 2 rho^k
    a = fma(ph.hgrav, rho0, a);
    a = fma(nuf[I], txx[ix(g, r, I - 1)] - txx[ix(g, r, I - 2)], a);
    a = fma(nuy, txy[ix(g, rp, I - 1)] - txy[ix(g, r, I - 1)], a);
    a = fma(-m.q4f[I], fma(sxp, up, -sxm * um), a);
    a = fma(-m.q4fy[I], fma(syp, vp, -sym * vm), a);
    const double gs = (p[ix(g, r, I - 1)] - p[ix(g, r, I)]) * m.ihxxf[I];
    const double ir2 = rcp_nr(den1[ix(g, r, I - 1)] + den1[ix(g, r, I)]);  // 1 / (2 rho^{k+1})
    double u = fma(adt2, a, rho0 * u0);
    if (k != 0) u = fma(bdt2, sxb[ix(g, r, I - 2)], u);
    u = fma(gdt2, gs, u);
    ux_out[ix(g, r, I - 1)] = u * ir2;
    sxa[ix(g, r, I - 2)] = a;
    if (sxg) sxg[ix(g, r, I - 2)] = gs;
  }
  // ---- uy at face (I, J - 1/2)
  {
    const double w0 = uy[ix(g, r, I)];
    const double sxm = mfx[ix(g, rm, I - 1)] + mfx[ix(g, r, I - 1)];
    const double sxp = mfx[ix(g, rm, I)] + mfx[ix(g, r, I)];
    const double um = uy[ix(g, r, I - 1)] + w0, up = w0 + uy[ix(g, r, I + 1)];
    const double f0 = mfy[ix(g, r, I)];
    const double sym = mfy[ix(g, rm, I)] + f0, syp = f0 + mfy[ix(g, rp, I)];
    const double vm = uy[ix(g, rm, I)] + w0, vp = w0 + uy[ix(g, rp, I)];
    double a = ifrcy[ix(g, r, I - 1)];
    a = fma(nuc[I], txy[ix(g, r, I)] - txy[ix(g, r, I - 1)], a);
    a = fma(nuy, tyy[ix(g, r, I - 1)] - tyy[ix(g, rm, I - 1)], a);
    a = fma(-m.q4c[I], fma(sxp, up, -sxm * um), a);
    a = fma(-g.q4y, fma(syp, vp, -sym * vm), a);
    const double gs = (p[ix(g, rm, I)] - p[ix(g, r, I)]) * g.ihy;
    const double rho0 = den0[ix(g, rm, I)] + den0[ix(g, r, I)];  // 2 rho^k
    const double ir2 = rcp_nr(den1[ix(g, rm, I)] + den1[ix(g, r, I)]);
    double u = fma(adt2, a, rho0 * w0);
    if (k != 0) u = fma(bdt2, syb[ix(g, r, I - 1)], u);
    u = fma(gdt2, gs, u);
    uy_out[ix(g, r, I)] = u * ir2;
    sya[ix(g, r, I - 1)] = a;
    if (syg) syg[ix(g, r, I - 1)] = gs;
  }
  // walls: impermeable, no-slip
  if (I == 1) {
    ux_out[ix(g, r, 0)] = 0.;
    uy_out[ix(g, r, 0)] = 0.;
  }
  if (I == g.nx) {
    ux_out[ix(g, r, g.nx)] = 0.;
    uy_out[ix(g, r, g.nx + 1)] = 0.;
  }
}

// ---------------------------------------------------------------------------
// momentum fluxes of the fused step, one per centre and corner
//   src/fluid/predict/ux.c:29-144, uy.c:29-130 (advective and diffusive
//   terms), txx.c:11-40, txy.c:13-50, tyy.c:10-38 (the stress components)
// The reference's advective term of ux at face i is a difference of products
// at the two neighbouring cell centres (along x) and corners (along y), and
// its diffusive term a difference of txx and txy at the same points; k_predict
// forms each product twice, once for each face it borders.  Here each point
// gets its flux once, scaled by 4 so that the 1/4 of the face averages
// moves into the face coefficient:
//   centre (I, J):     Pxx = 4 nu txx - (mfx_I + mfx_I+1) (ux_I + ux_I+1)
//                      Pyy = 4 nu tyy - (mfy_J-1/2 + mfy_J+1/2) (uy_J-1/2 + uy_J+1/2)
//   corner (I, J-1/2): Pxy = 4 nu txy - r_I (mfy_I-1 + mfy_I) (ux_J-1 + ux_J)
//                      Pyx = 4 nu txy - (mfx_J-1 + mfx_J) (uy_I-1 + uy_I)
// (mfx, mfy the mass fluxes, r_I = HXXC / HXXF(I) the metric ratio of the
// reference's y advection of ux).  k_predict_mf then adds, with nu / H =
// 4 nu (0.25 / H), the reference's diffusion minus advection
//   ux face I:    0.25 / HXXF(I) (Pxx_I - Pxx_I-1) + 0.25 / hy (Pxy_J+1/2 - Pxy_J-1/2)
//   uy face J-1/2: 0.25 / HXXC(I) (Pyx_I+1 - Pyx_I) + 0.25 / hy (Pyy_J - Pyy_J-1)
// FP64 operations per cell: 29 here (27 with the viscosities pre-scaled)
// and 33 in k_predict_mf (with the Poisson face values it also writes)
// against 16 + 61 for k_stress + k_predict.
// STRESS 1: also txy at the wall columns I = 1, nx + 1 (what the wall-stress
// log reads, src/logging/stress.c); 2: the whole of txx, txy, tyy, in the
// reference's form.  SCALED: visux, visuy come times nuy2 and nuy4
// (k_props<..., true>), so 4 nu txy = sx du + sy dw hy / (2 HXXF) and
// 4 nu tyy = sy dw: two FP64 multiplies per cell fewer (STRESS 0 or 1)
// thread (I, J): I = 1..nx+1 handles the corner (I, J - 1/2) and, for I <= nx,
// the centre (I, J)
// ---------------------------------------------------------------------------
// HOW the momentum kernels run a cell (chosen in stencil_how): both parts of
// it (the corner and the centre; the ux and the uy face) in one thread, shared
// with the integer pipes; one part a thread, the blocks of even and odd row
// index taking one each, so that a warp's chain of instructions and loads is
// half as long, shared or on the FP64 unit alone
enum MomHow { kMomWhole, kMomSplitInt, kMomSplit };
struct MomIn {
  double u0, us, u1, w0, ww, w1;        // ux at face I: row J, row J-1; at face I+1.  uy: cell I, I-1; row J+1/2
  double vx0, vxs, vx1, vy0, vyw, vyn;  // viscosities, likewise
  double mx0, mxs, mx1, my0, myw, my1;  // mass fluxes, likewise
  double rq, c2, c4;
};
struct MomOut {
  double xx, yy, xy, yx;
};

// A step whose ux is zero everywhere (fluid at rest, or moving along y only)
// has zeros where the integer forms of the momentum kernels take none, in
// every cell: decide_dt says so (kScStill), and such a step runs on the FP64
// unit from the start.  2048 x 1024 at rest, a step: 2185 us with the integer
// forms tried first, 1531 us without; 509 x 256 220 and 179 us.  Both paths
// use the cell's loaded inputs, so that the loads stay ahead of the branch,
// and take the registers of four blocks an SM.  A step in motion, 1000 x 512
// and 509 x 256: without the branch 472 and 207 us (five blocks), with it 472
// and 212 us (five), 467 and 205 us (four); the zeros looked for in each
// cell's own values, 483 and 211 us (five).
__device__ __forceinline__ bool still(const double *__restrict__ sc) { return __double2hiint(sc[kScStill]) != 0; }

// the four fluxes of one thread (PART 1: the corner's two, 2: the centre's); returns whether an integer form gave up.
// Of the 27 FP64 operations (SCALED) the four sum-and-difference pairs of the
// velocities and four of the products run on the integer pipes.  2048 x 1024
// swarm, one launch: 110.6 us all in FP64 (FP64 unit 85% busy); 69.1 us with
// a fifth product on the integer side (integer pipes 90%, FP64 73%), 73.6 us
// with one sum more; 65.9 us as it stands at five blocks an SM (89%, 82%), 64.1
// us at four (94%, 85%).
template <bool INT, bool SCALED, int PART = 0>
__device__ __forceinline__ bool momflux_cell(const Fp64 &f, const MomIn &in, const Phys &ph, MomOut &o) {
  Fp64Int<INT> q(f);
  if (PART != 2) {  // corner
    double su, du, sw, dw;
    q.template addsub<true>(in.u0, in.us, su, du);  // zero along the walls
    q.addsub(in.w0, in.ww, sw, dw);
    const double sx = f.add(in.vxs, in.vx0), sy = f.add(in.vyw, in.vy0);
    const double t4 = fma(sx, SCALED ? du : f.mul(du, f.reg(ph.nuy2)), q.mul(sy, q.mul(dw, in.c2)));  // 4 nu txy
    const double fy = f.add(in.myw, in.my0), fx = f.add(in.mxs, in.mx0);
    o.xy = fma(-q.mul(in.rq, fy), su, t4);
    o.yx = fma(-fx, sw, t4);
  }
  if (PART != 1) {  // centre
    double su, du, sw, dw;
    q.addsub(in.u1, in.u0, su, du);
    q.addsub(in.w1, in.w0, sw, dw);
    const double sx = f.add(in.vx0, in.vx1), sy = f.add(in.vy0, in.vyn);
    o.xx = fma(-f.add(in.mx0, in.mx1), su, f.mul(sx, q.mul(du, in.c4)));
    o.yy = fma(-f.add(in.my0, in.my1), sw, f.mul(sy, SCALED ? dw : f.mul(dw, f.reg(ph.nuy4))));
  }
  return INT && q.bad != 0;
}

template <int STRESS, bool SCALED, int HOW>
__global__ void __launch_bounds__(BX *BY, SCALED && HOW == kMomWhole ? 4 : 1)
    k_momflux(Grid g, Metrics m, Phys ph0, const double *__restrict__ sc, const double *__restrict__ ux,
              const double *__restrict__ uy,
              const double *__restrict__ visux, const double *__restrict__ visuy, const double *__restrict__ mfx,
              const double *__restrict__ mfy, double *__restrict__ pxx, double *__restrict__ pyy,
              double *__restrict__ pxy, double *__restrict__ pyx, double *__restrict__ txx, double *__restrict__ txy,
              double *__restrict__ tyy) {
  pdl_entry();
  sc += (size_t)blockIdx.z * (kScalars);
  const Phys ph = zphys(g, ph0);
  static_assert(!(SCALED && STRESS == 2), "the reference-form stresses take unscaled viscosities");
  const double *__restrict__ c4nuc = SCALED ? m.c4nucs : m.c4nuc + (size_t)blockIdx.z * g.cm;
  const double *__restrict__ c2nuf = SCALED ? m.c2nufs : m.c2nuf + (size_t)blockIdx.z * g.cm;
  const int I = blockIdx.x * blockDim.x + threadIdx.x + 1;
  // the unscaled forms (full-sync steps) run whole, on the FP64 unit alone
  constexpr bool SPLIT = SCALED && HOW != kMomWhole, INT = SCALED && HOW != kMomSplit;
  const bool corner = !SPLIT || !(blockIdx.y & 1);
  const int J = (SPLIT ? blockIdx.y >> 1 : blockIdx.y) * blockDim.y + threadIdx.y + 1;
  if (I > g.nx + 1 || J > g.ny) return;
  const Fp64 f(I);
  const int zr = blockIdx.z * g.ny;  // first row of this case
  const int r = J - 1 + zr, rm = wrap(J - 1, g.ny) + zr, rp = wrap(J + 1, g.ny) + zr;
  const bool centre = I <= g.nx && (!SPLIT || !corner);
  // centre (I, J); the threads of the last face have none and take the column before
  const int Ic = I <= g.nx ? I : I - 2;
  auto load = [&](int r, int rm, int rp) {
    MomIn in;
    in.u0 = ux[ix(g, r, I - 1)];  // ux at face I, row J
    in.vx0 = visux[ix(g, r, I - 1)];
    in.w0 = uy[ix(g, r, I)];  // uy of cell I at J - 1/2
    in.vy0 = visuy[ix(g, r, I)];
    in.mx0 = mfx[ix(g, r, I - 1)];
    in.my0 = mfy[ix(g, r, I)];
    // corner (I, J - 1/2)
    in.us = ux[ix(g, rm, I - 1)];
    in.ww = uy[ix(g, r, I - 1)];
    in.vxs = visux[ix(g, rm, I - 1)];
    in.vyw = visuy[ix(g, r, I - 1)];
    in.mxs = mfx[ix(g, rm, I - 1)];
    in.myw = mfy[ix(g, r, I - 1)];
    in.rq = m.rq[I];
    in.c2 = c2nuf[I];
    // centre
    in.u1 = ux[ix(g, r, Ic)];
    in.w1 = uy[ix(g, rp, Ic)];
    in.vx1 = visux[ix(g, r, Ic)];
    in.vyn = visuy[ix(g, rp, I)];
    in.mx1 = mfx[ix(g, r, Ic)];
    in.my1 = mfy[ix(g, rp, I)];
    in.c4 = c4nuc[Ic];
    return in;
  };
  const bool at_rest = INT && !SPLIT && still(sc);
  MomIn in = load(r, rm, rp);
  MomOut o;
  auto cell = [&](auto part) {
    bool redo = at_rest;
    if (!redo && (redo = momflux_cell<INT, SCALED, part>(f, in, ph, o))) in = load(reread(r), reread(rm), reread(rp));
    if (redo) momflux_cell<false, SCALED, part>(f, in, ph, o);
  };
  if (!SPLIT)
    cell(std::integral_constant<int, 0>());
  else if (corner)
    cell(std::integral_constant<int, 1>());
  else
    cell(std::integral_constant<int, 2>());
  if (corner) {
    pxy[ix(g, r, I - 1)] = o.xy;
    pyx[ix(g, r, I - 1)] = o.yx;
  }
  if (corner && (STRESS == 2 || (STRESS == 1 && (I == 1 || I == g.nx + 1)))) {
    // txy = 0.5 (mu_s + mu_n) du/dy + 0.5 (mu_w + mu_e) dv/dx
    if (!SPLIT) in = load(reread(r), reread(rm), reread(rp));
    const double sx = in.vxs + in.vx0, sy = in.vyw + in.vy0, du = in.u0 - in.us, dw = in.w0 - in.ww;
    txy[ix(g, r, I - 1)] = SCALED ? fma(sx, du * (g.hihy * ph.inuy2), sy * (dw * (m.hihxxf[I] * ph.inuy4)))
                                  : fma(sx, du * g.hihy, sy * (dw * m.hihxxf[I]));
  }
  if (centre) {
    pxx[ix(g, r, I - 1)] = o.xx;
    pyy[ix(g, r, I - 1)] = o.yy;
    if (STRESS == 2) {
      txx[ix(g, r, I - 1)] = (in.vx0 + in.vx1) * ((in.u1 - in.u0) * m.ihxxc[I]);
      tyy[ix(g, r, I - 1)] = (in.vy0 + in.vyn) * ((in.w1 - in.w0) * g.ihy);
    }
  }
}

// ---------------------------------------------------------------------------
// momentum right-hand sides and the RK predictor of the fused step, from the
// fluxes of k_momflux (the terms of k_predict, same discretisation)
//   src/fluid/predict/ux.c:146-273, uy.c:132-251, main.c:9-80
// Also stores, at both faces, e grad psi_old with e = rho_ref / rho^{k+1} - 1
// and psi_old the potential of the previous substage: the variable-density
// term of the Poisson right-hand side (src/fluid/compute_potential.c:
// 285-363) and of the velocity correction (src/fluid/correct_velocity/ux.c:
// 18-66, uy.c:17-64) is the same face quantity, so both read it from here.
// CACHED: 2 rho^k at the faces is the 2 rho^{k+1} the previous substage's
// predictor formed (srx, sry, which this one overwrites with its own), and
// psi_old's differences across the faces are the ones the previous
// substage's correction formed (dpx, dpy); else both come from den0 and
// psio (first substage of a step whose state may be new).  The same values
// either way.
// thread (I, J): I = 1..nx handles the ux face I (I >= 2) and the uy face
// (I, J - 1/2)
// ---------------------------------------------------------------------------
struct PredIn {
  double u0, frc, rho0, dps;  // velocity, surface tension, 2 rho^k, psi_old's difference across the face
  double pd1, pd0, po1, po0;  // fluxes either side of the face, along it and across
  double r1a, r1b, p0, p1, sb;  // rho^{k+1} and p of the two cells, the last substage's right-hand side
  double cd, co, gp, rp, pa, pd;
};
struct PredOut {
  double rho1, u, a, e, q;
};

// one face; returns whether an integer form gave up.  The FP64 unit keeps the
// fused multiply-adds and the pressure difference (zero everywhere in a first
// step, which the integer form would leave to it).  2048 x 1024 swarm, one
// launch: 137.4 us all in FP64; with the integer forms 119.8 us, the loads of
// the second face then exposed (warps waiting on global memory 6.5 of 9.6
// cycles an issue); 106 us with those loads in flight during the first face
// (yb); 99.7 us at five blocks an SM and the pressure difference in FP64, 97.4
// us at four with still()'s branch.
template <bool INT, bool GRAV>
__device__ __forceinline__ bool predict_face(const Fp64 &f, const PredIn &in, double hgrav, double adt2, double bdt2,
                                             int k, PredOut &o) {
  Fp64Int<INT> n(f);
  double a = in.frc;
  if (GRAV) a = fma(hgrav, in.rho0, a);
  a = fma(in.cd, n.sub(in.pd1, in.pd0), a);
  a = fma(in.co, n.sub(in.po1, in.po0), a);
  o.rho1 = n.addp(in.r1a, in.r1b);  // 2 rho^{k+1}
  const double ir2 = rcp_nr(o.rho1, f);
  double u = fma(adt2, a, n.mul(in.rho0, in.u0));
  if (k != 0) u = fma(bdt2, in.sb, u);
  u = fma(in.gp, f.sub(in.p0, in.p1), u);
  o.u = n.mul(u, ir2);
  o.a = a;
  o.e = n.mulz(fma(in.rp, ir2, -in.pa), in.dps);
  o.q = fma(in.pd, o.u, o.e);
  return INT && n.bad != 0;
}

template <bool CACHED, int HOW>
__global__ void __launch_bounds__(BX *BY, HOW == kMomWhole ? 4 : 1)
    k_predict_mf(Grid g, Metrics m, Phys ph0, const double *__restrict__ sc, int k, const double *__restrict__ ux,
                 const double *__restrict__ uy, double *__restrict__ ux_out, double *__restrict__ uy_out,
                 const double *__restrict__ pxx, const double *__restrict__ pyy, const double *__restrict__ pxy,
                 const double *__restrict__ pyx, const double *__restrict__ p, const double *__restrict__ ifrcx,
                 const double *__restrict__ ifrcy, const double *__restrict__ den0, const double *__restrict__ den1,
                 const double *__restrict__ psio, double *__restrict__ sxa, const double *__restrict__ sxb,
                 double *__restrict__ sya, const double *__restrict__ syb, double *__restrict__ egx,
                 double *__restrict__ egy, const double *__restrict__ coltab, double *__restrict__ qx,
                 double *__restrict__ qy, double *__restrict__ srx, double *__restrict__ sry,
                 const double *__restrict__ dpx, const double *__restrict__ dpy) {
  pdl_entry();
  sc += (size_t)blockIdx.z * (kScalars);
  const double *__restrict__ gx = coltab + ((size_t)blockIdx.z * 3 * kColTabs + ct_gdt2x(k)) * g.ct;
  // the Poisson right-hand side's face values q = pd u* + pa e grad psi_old
  // (k_poisson_fwd<W, true> takes their differences across each cell)
  const int I = blockIdx.x * blockDim.x + threadIdx.x + 1;
  constexpr bool WHOLE = HOW == kMomWhole, INT = HOW != kMomSplit;
  const bool do_x = WHOLE || !(blockIdx.y & 1), do_y = WHOLE || (blockIdx.y & 1);
  const int J = (WHOLE ? blockIdx.y : blockIdx.y >> 1) * blockDim.y + threadIdx.y + 1;
  if (I > g.nx || J > g.ny) return;
  const Fp64 f(I);
  const int zr = blockIdx.z * g.ny;  // first row of this case
  const int r = J - 1 + zr, rm = wrap(J - 1, g.ny) + zr, rp = wrap(J + 1, g.ny) + zr;
  // the update is carried as 2u with 2 alpha dt, ... and 1 / (2 rho_face):
  // powers of two, so every rounding is the one of the plain form; the
  // pressure term's 2 gamma dt / H comes per column (gx) or per case
  const double adt2 = sc[sc_adt2(k)], bdt2 = sc[sc_bdt2(k)];
  const Phys ph = zphys(g, ph0);
  // e grad psi_old is stored times the Poisson factor pax (x faces) or pay
  // (y faces): e pa = (2 rho_ref pa) / (2 rho) - pa
  const double rpx = sc[sc_rpx(k)], pax = sc[sc_pax(k)];
  const double q4y = f.reg(g.q4y), hgrav = f.reg(ph.hgrav);
  __shared__ double yb[WHOLE ? 11 : 1][BX * BY];
  const int tid = threadIdx.y * blockDim.x + threadIdx.x;
  if (WHOLE) {
    async_copy(&yb[0][tid], uy + ix(g, r, I));
    async_copy(&yb[1][tid], ifrcy + ix(g, r, I - 1));
    async_copy(&yb[2][tid], pyx + ix(g, r, I));
    async_copy(&yb[3][tid], pyx + ix(g, r, I - 1));
    async_copy(&yb[4][tid], pyy + ix(g, r, I - 1));
    async_copy(&yb[5][tid], pyy + ix(g, rm, I - 1));
    async_copy(&yb[6][tid], den1 + ix(g, rm, I));
    async_copy(&yb[7][tid], p + ix(g, rm, I));
    if (k != 0) async_copy(&yb[8][tid], syb + ix(g, r, I - 1));
    if (CACHED) {
      async_copy(&yb[9][tid], sry + ix(g, r, I));
      async_copy(&yb[10][tid], dpy + ix(g, r, I));
    }
  }
  const bool at_rest = INT && still(sc);
  const double ps0 = CACHED && I != 1 && I != g.nx ? 0. : psio[ix(g, r, I)];
  // ---- ux at face I
  if (do_x && I >= 2) {
    auto load = [&](int r, int rm, int rp) {
      PredIn in;
      in.u0 = ux[ix(g, r, I - 1)];
      in.frc = ifrcx[ix(g, r, I - 2)];
      in.pd1 = pxx[ix(g, r, I - 1)], in.pd0 = pxx[ix(g, r, I - 2)];
      in.po1 = pxy[ix(g, rp, I - 1)], in.po0 = pxy[ix(g, r, I - 1)];
      in.r1a = den1[ix(g, r, I - 1)], in.r1b = den1[ix(g, r, I)];
      in.p0 = p[ix(g, r, I - 1)], in.p1 = p[ix(g, r, I)];
      in.sb = k != 0 ? sxb[ix(g, r, I - 2)] : 0.;
      in.rho0 = CACHED ? srx[ix(g, r, I - 1)] : f.add(den0[ix(g, r, I - 1)], den0[ix(g, r, I)]);  // 2 rho^k
      in.dps = CACHED ? dpx[ix(g, r, I - 1)] : f.sub(ps0, psio[ix(g, r, I - 1)]);
      in.cd = m.q4f[I], in.co = q4y, in.gp = gx[I], in.rp = rpx, in.pa = pax, in.pd = sc[sc_pdx(k)];
      return in;
    };
    PredOut o;
    PredIn in = load(r, rm, rp);
    bool redo = INT && at_rest;
    if (!redo && (redo = predict_face<INT, true>(f, in, hgrav, adt2, bdt2, k, o)))
      in = load(reread(r), reread(rm), reread(rp));
    if (redo) predict_face<false, true>(f, in, hgrav, adt2, bdt2, k, o);
    srx[ix(g, r, I - 1)] = o.rho1;
    ux_out[ix(g, r, I - 1)] = o.u;
    sxa[ix(g, r, I - 2)] = o.a;
    egx[ix(g, r, I - 1)] = o.e;
    qx[ix(g, r, I - 1)] = o.q;
  }
  // ---- uy at face (I, J - 1/2)
  if (do_y) {
    auto coefs = [&](PredIn &in) {
      in.cd = m.q4c[I], in.co = q4y, in.gp = sc[sc_gdt2y(k)], in.rp = sc[sc_rpy(k)], in.pa = sc[sc_pay(k)],
      in.pd = sc[sc_pdy(k)];
    };
    auto load = [&](int r, int rm) {
      PredIn in;
      in.u0 = uy[ix(g, r, I)], in.frc = ifrcy[ix(g, r, I - 1)];
      in.pd1 = pyx[ix(g, r, I)], in.pd0 = pyx[ix(g, r, I - 1)];
      in.po1 = pyy[ix(g, r, I - 1)], in.po0 = pyy[ix(g, rm, I - 1)];
      in.r1a = den1[ix(g, rm, I)], in.r1b = den1[ix(g, r, I)];
      in.p0 = p[ix(g, rm, I)], in.p1 = p[ix(g, r, I)];
      in.sb = k != 0 ? syb[ix(g, r, I - 1)] : 0.;
      in.rho0 = CACHED ? sry[ix(g, r, I)] : f.add(den0[ix(g, rm, I)], den0[ix(g, r, I)]);  // 2 rho^k
      in.dps = CACHED ? dpy[ix(g, r, I)] : f.sub(psio[ix(g, r, I)], psio[ix(g, rm, I)]);
      coefs(in);
      return in;
    };
    PredOut o;
    PredIn in;
    if (WHOLE) {
      async_wait();
      in.u0 = yb[0][tid], in.frc = yb[1][tid];
      in.pd1 = yb[2][tid], in.pd0 = yb[3][tid];
      in.po1 = yb[4][tid], in.po0 = yb[5][tid];
      in.r1a = yb[6][tid], in.r1b = den1[ix(g, r, I)];
      in.p0 = yb[7][tid], in.p1 = p[ix(g, r, I)];
      in.sb = k != 0 ? yb[8][tid] : 0.;
      in.rho0 = CACHED ? yb[9][tid] : f.add(den0[ix(g, rm, I)], den0[ix(g, r, I)]);  // 2 rho^k
      in.dps = CACHED ? yb[10][tid] : f.sub(ps0, psio[ix(g, rm, I)]);
      coefs(in);
    } else {
      in = load(r, rm);
    }
    bool redo = INT && at_rest;
    if (!redo && (redo = predict_face<INT, false>(f, in, hgrav, adt2, bdt2, k, o))) in = load(reread(r), reread(rm));
    if (redo) predict_face<false, false>(f, in, hgrav, adt2, bdt2, k, o);
    sry[ix(g, r, I)] = o.rho1;
    uy_out[ix(g, r, I)] = o.u;
    sya[ix(g, r, I - 1)] = o.a;
    egy[ix(g, r, I)] = o.e;
    qy[ix(g, r, I)] = o.q;
  }
  // walls: impermeable, no-slip; the wall faces' e grad psi_old (zero for a
  // Neumann psi_old, computed as the reference does)
  if (do_x && I == 1) {
    ux_out[ix(g, r, 0)] = 0.;
    uy_out[ix(g, r, 0)] = 0.;
    const double e = fma(rpx, rcp_nr(den1[ix(g, r, 0)] + den1[ix(g, r, 1)]), -pax) * (ps0 - psio[ix(g, r, 0)]);
    egx[ix(g, r, 0)] = e;
    qx[ix(g, r, 0)] = fma(sc[sc_pdx(k)], 0., e);
  }
  if (do_x && I == g.nx) {
    ux_out[ix(g, r, g.nx)] = 0.;
    uy_out[ix(g, r, g.nx + 1)] = 0.;
    const double e =
        fma(rpx, rcp_nr(den1[ix(g, r, g.nx)] + den1[ix(g, r, g.nx + 1)]), -pax) * (psio[ix(g, r, g.nx + 1)] - ps0);
    egx[ix(g, r, g.nx)] = e;
    qx[ix(g, r, g.nx)] = fma(sc[sc_pdx(k)], 0., e);
  }
}

// ---------------------------------------------------------------------------
// Poisson solve for the scalar potential (src/fluid/compute_potential.c)
//
// The reference diagonalises the constant-coefficient operator with a DCT
// along x and solves one periodic tridiagonal system along y per x
// wavenumber.  Here the same discrete operator is diagonalised by a real DFT
// along the periodic y direction and one (non-periodic, Neumann-ended)
// tridiagonal system along x is solved per y wavenumber.
//   1. k_poisson_fwd: right-hand side of src/fluid/compute_potential.c:
//      285-363 for a tile of W columns,
//        rhs = rho_ref/dt_new div u* - dt_old/dt_new div((rho_ref/rho - 1) grad psi_old)
//      (the face values of (rho_ref/rho - 1) grad psi_old come from k_predict_mf,
//      already times their Poisson coefficient; in the fused step the
//      predictor also adds the u* term at each face, so the transform only
//      differences the sums)
//      with div and the face differences in the JD = H hy form, packed two
//      reals per complex, a mixed radix-4/2 Stockham FFT of length ny/2 in
//      shared memory and the real-to-complex split; spectrum [I][m]
//   2. k_poisson_tdm: tridiagonal solves along x (warp-parallel scan)
//   3. k_poisson_inv: inverse of step 1, psi and its Neumann ghosts
// The 1 / ny of the inverse DFT and the 1/2 of the real split are folded
// into the right-hand-side coefficients.
// ---------------------------------------------------------------------------

// -i z (forward) or +i z (inverse)
__device__ __forceinline__ double2 rot(double2 z, bool inverse) {
  return inverse ? make_double2(-z.y, z.x) : make_double2(z.y, -z.x);
}

// One untwiddled radix-8 butterfly, xr[0], xr[q], .. xr[7 q] into yr[0..7];
// returns whether an integer form gave up.
//   X_2m = DFT4(v_q + v_q+4)_m, X_2m+1 = DFT4((v_q - v_q+4) W8^q)_m; the
//   1/sqrt(2) of W8 and W8^3 rides in the odd half's last FMAs: 52 FP64
//   operations for 8 points, where a radix-2 stage and a twiddled radix-4
//   stage take 64 for the same three levels
// INT: 24 of the 52, the sums and differences of the first level and of the
// even half's second, run on the integer pipes.
template <bool INT>
__device__ __forceinline__ bool radix8(const Fp64 &f, const double2 *xr, double2 *yr, int q, double c8, bool inverse) {
  Fp64Int<INT> n(f);
  double2 a[4], b[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) n.caddsub(xr[i * q], xr[(i + 4) * q], a[i], b[i]);
  // even outputs: DFT4 of a
  double2 e0, e1, e2, e3;
  n.caddsub(a[0], a[2], e0, e1);
  n.caddsub(a[1], a[3], e2, e3);
  const double2 re3 = rot(e3, inverse);
  yr[0] = f.cadd(e0, e2);
  yr[2] = f.cadd(e1, re3);
  yr[4] = f.csub(e0, e2);
  yr[6] = f.csub(e1, re3);
  // odd outputs: t1 = b1 W8 = c8 P1, t2 = b2 W8^2 (a rotation), t3 = b3 W8^3 = c8 P3
  const double2 P1 = inverse ? make_double2(f.sub(b[1].x, b[1].y), f.add(b[1].x, b[1].y))
                             : make_double2(f.add(b[1].x, b[1].y), f.sub(b[1].y, b[1].x));
  const double2 P3 = inverse ? make_double2(-f.add(b[3].x, b[3].y), f.sub(b[3].x, b[3].y))
                             : make_double2(f.sub(b[3].y, b[3].x), -f.add(b[3].x, b[3].y));
  const double2 t2 = rot(b[2], inverse);
  const double2 A0 = f.cadd(b[0], t2), A1 = f.csub(b[0], t2);
  const double2 E = f.cadd(P1, P3), D = f.csub(P1, P3);  // t1 + t3 = c8 E, t1 - t3 = c8 D
  const double2 rD = rot(D, inverse);
  yr[1] = make_double2(fma(c8, E.x, A0.x), fma(c8, E.y, A0.y));
  yr[3] = make_double2(fma(c8, rD.x, A1.x), fma(c8, rD.y, A1.y));
  yr[5] = make_double2(fma(-c8, E.x, A0.x), fma(-c8, E.y, A0.y));
  yr[7] = make_double2(fma(-c8, rD.x, A1.x), fma(-c8, rD.y, A1.y));
  return INT && n.bad != 0;
}

// One radix-4 butterfly, xr[0], xr[q], xr[2 q], xr[3 q] into yr[0], yr[s],
// yr[2 s], yr[3 s], the inputs times 1, wm[e], wm[2 e], wm[3 e] (TWIDDLE);
// returns whether an integer form gave up.
//   a0 = v0 + w2 v2 and a2 = w1 v1 + w3 v3 with the products folded into
//   FMAs, a1 = 2 v0 - a0 and a3 = 2 (w1 v1) - a2: 24 FP64 operations per
//   butterfly instead of 28 (cmul, then add and subtract)
// INT: the eight closing sums and differences and two products run on the
// integer pipes (without twiddles, the eight opening ones).  2048 x 1024, one
// launch, FP64 alone -> shared: k_poisson_fwd 70.5 -> 55.3 us, k_poisson_inv
// 58.0 -> 46.3 us (56.9 and 46.6 with the two products left in FP64; 60.8 and
// 51.5 at three blocks an SM, 60.8 and 46.4 at five).
template <bool INT, bool TWIDDLE>
__device__ __forceinline__ bool radix4(const Fp64 &f, const double2 *xr, double2 *yr, int q, int s,
                                       const double2 *__restrict__ wm, int e, double two, bool inverse) {
  Fp64Int<INT> n(f);
  const double2 v0 = xr[0], v1 = xr[q], v2 = xr[2 * q], v3 = xr[3 * q];
  if (TWIDDLE) {
    const double2 w1 = wm[e], w2 = wm[2 * e], w3 = wm[3 * e];
    const double2 a0 = make_double2(fma(w2.x, v2.x, fma(-w2.y, v2.y, v0.x)), fma(w2.x, v2.y, fma(w2.y, v2.x, v0.y)));
    const double2 a1 = make_double2(fma(two, v0.x, -a0.x), fma(two, v0.y, -a0.y));
    const double2 t1 = make_double2(fma(v1.x, w1.x, n.mulz(-v1.y, w1.y)), fma(v1.x, w1.y, n.mulz(v1.y, w1.x)));
    const double2 a2 = make_double2(fma(w3.x, v3.x, fma(-w3.y, v3.y, t1.x)), fma(w3.x, v3.y, fma(w3.y, v3.x, t1.y)));
    const double2 a3 = make_double2(fma(two, t1.x, -a2.x), fma(two, t1.y, -a2.y));
    const double2 r3 = rot(a3, inverse);
    n.caddsub(a0, a2, yr[0], yr[2 * s]);
    n.caddsub(a1, r3, yr[s], yr[3 * s]);
  } else {
    double2 a0, a1, a2, a3;
    n.caddsub(v0, v2, a0, a1);
    n.caddsub(v1, v3, a2, a3);
    const double2 r3 = rot(a3, inverse);
    yr[0] = f.cadd(a0, a2);
    yr[s] = f.cadd(a1, r3);
    yr[2 * s] = f.csub(a0, a2);
    yr[3 * s] = f.csub(a1, r3);
  }
  return INT && n.bad != 0;
}

// The same butterflies with one thread per component and output, for launches
// of a few warps, whose time is one thread's chain of FP64 instructions (65
// cycles each): 4 in turn instead of 52 (radix 8, 16 lanes), 6 instead of 24
// (radix 4 with twiddles, 8 lanes), 2 instead of 16 (without).  Every value
// comes from the operation that radix8 and radix4 form it with.  Lanes of a
// butterfly are l = 0, 1, ..; x is the value a lane holds, c the component it
// belongs to, flip() a sign change where `neg` is set.  rot(z) has component c
// from z's other one, negated where turn(c) is set.
__device__ __forceinline__ double flip(double x, bool neg) {
  return __hiloint2double(__double2hiint(x) ^ (neg ? (int)0x80000000 : 0), __double2loint(x));
}
__device__ __forceinline__ double part(double2 z, int c) { return c ? z.y : z.x; }
__device__ __forceinline__ void put(double2 *z, int c, double x) { reinterpret_cast<double *>(z)[c] = x; }

__device__ __forceinline__ void radix8_lanes(const Fp64 &f, const double2 *xr, double2 *yr, int q8, double c8,
                                             bool inverse, int l, bool store) {
  const unsigned all = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int c = l & 1, q = (l >> 1) & 3;
  const bool odd = l >> 3;  // the lanes of b, else of a
  auto turn = [inverse](int c) { return (c == 1) != inverse; };
  // a_q = v_q + v_q+4, b_q = v_q - v_q+4
  double x = fma(flip(part(xr[(q + 4) * q8], c), odd), f.one, part(xr[q * q8], c));
  // a: e0 = a0 + a2, e2 = a1 + a3, e1 = a0 - a2, e3 = a1 - a3 in lanes q = 0 .. 3;
  // b: A0 = b0 + rot b2, P1, A1 = b0 - rot b2 (component 1 - c), P3
  const bool hi = q >= 2;
  double o = __shfl_sync(all, x, lane ^ (!odd ? 4 : ((q & 1) ? 1 : 5)));
  bool nx, no, nr = false;  // signs of x, o and the sum
  if (!odd) {
    nx = hi, no = false;
  } else if (q == 3) {  // forward (y - x, -(x + y)), inverse (-(x + y), x - y)
    nx = !turn(c), no = false, nr = turn(c);
  } else if (q == 2) {
    nx = !turn(1 - c), no = false;
  } else {
    nx = false, no = turn(c);
  }
  x = flip(fma(flip(x, nx), f.one, flip(o, no)), nr);
  // a: X0 = e0 + e2, X4 = e0 - e2, X2 = e1 + rot e3, X6 = e1 - rot e3 (component 1 - c);
  // b: E = P1 + P3 in lanes q = 1, D = P1 - P3 in lanes q = 3
  o = __shfl_sync(all, x, lane ^ (odd ? 4 : (hi ? 3 : 2)));
  if (!odd) {
    nx = q == 1 || (q == 3 && !turn(1 - c));
    no = q == 2 && turn(c);
  } else {
    nx = q == 3, no = false;
  }
  const double y = fma(flip(x, nx), f.one, flip(o, no));
  if (!odd || (q & 1)) x = y;
  // b: X1, X5 = A0 +- c8 E, X3, X7 = A1 +- c8 rot D
  o = __shfl_sync(all, x, lane ^ 2);
  const int oc = hi && (odd || q == 3) ? 1 - c : c;
  if (odd) {
    const double m = (q & 1) ? x : o, a = (q & 1) ? o : x;
    x = fma(flip(c8, q & 1), flip(m, hi && turn(oc)), a);
  }
  const int at = odd ? (q == 0 ? 1 : (q == 1 ? 5 : (q == 2 ? 3 : 7))) : (q == 0 ? 0 : (q == 1 ? 4 : (q == 2 ? 2 : 6)));
  if (store) put(yr + at, oc, x);
}

template <bool TWIDDLE>
__device__ __forceinline__ void radix4_lanes(const Fp64 &f, const double2 *xr, double2 *yr, int q, int s,
                                             const double2 *__restrict__ wm, int e, double two, bool inverse, int l,
                                             bool store) {
  const int lane = threadIdx.x & 31;
  const int c = l & 1;
  const bool sub = l & 2, h = l & 4;  // the lanes of a1, a3 (else a0, a2); of a2, a3 (else a0, a1)
  const double2 vb = xr[h ? q : 0], vd = xr[h ? 3 * q : 2 * q];
  double x;
  if (TWIDDLE) {
    const double2 w = wm[(h ? 3 : 2) * e];
    double b = part(vb, c);
    if (h) {
      const double2 w1 = wm[e];
      b = fma(vb.x, part(w1, c), f.mul(flip(vb.y, c == 0), part(w1, 1 - c)));
    }
    const double a = fma(w.x, part(vd, c), fma(flip(w.y, c == 0), part(vd, 1 - c), b));
    x = fma(two, b, -a);
    if (!sub) x = a;
  } else {
    x = fma(flip(part(vd, c), sub), f.one, part(vb, c));
  }
  // X0 = a0 + a2, X1 = a1 + rot a3, X2 = a0 - a2, X3 = a1 - rot a3 (component 1 - c)
  const double o = __shfl_sync(0xffffffffu, x, lane ^ (sub ? 5 : 4));
  const int oc = h && sub ? 1 - c : c;
  const bool turned = sub && ((oc == 1) != inverse);
  const double a = h ? o : x, r = flip(h ? x : o, turned != h);
  x = fma(r, f.one, a);
  if (store) put(yr + ((sub ? 1 : 0) + (h ? 2 : 0)) * s, oc, x);
}

// Stockham FFT (radix 4, one radix-8 stage first when log2 M is odd) of the
// first `cols` of W rows of length M in shared memory.  Returns the buffer
// holding the result.
// tw: the twiddle buffer, exp(-2 pi i m / 2M) for m = 0..M, then W_M^e for
// e < M, then their conjugates (the inverse's): one load per twiddle.
// HOW: a thread's butterflies on the FP64 unit (kFftPlain; kFftShort with the
// registers of five blocks an SM, for launches that have them), shared with
// the integer pipes (kFftInt), or spread over lanes (kFftLanes).
enum FftHow { kFftPlain, kFftInt, kFftLanes, kFftShort };
template <int W, int HOW>
__device__ double2 *fft_rows(double2 *x, double2 *y, int M, const double2 *__restrict__ tw, bool inverse, const Fp64 &f,
                             int cols) {
  constexpr bool INT = HOW == kFftInt;
  const double two = f.reg(2.);
  const double2 *__restrict__ wm = tw + (M + 1) + (inverse ? M : 0);
  int Ns = 1;
  if ((__ffs(M) - 1) & 1) {  // log2 M odd (M >= 8)
    const double c8 = f.reg(0.70710678118654752440);
    const int q8 = M >> 3;
    // lanes: whole warps take part in the exchanges, the last ones as copies
    for (int t = threadIdx.x; HOW == kFftLanes && t < ((16 * cols * q8 + 31) & ~31); t += blockDim.x) {
      const bool in = t < 16 * cols * q8;
      const int b = in ? t >> 4 : 0, c = b / q8, j = b - c * q8;
      radix8_lanes(f, x + c * M + j, y + c * M + 8 * j, q8, c8, inverse, t & 15, in);
    }
    for (int t = threadIdx.x; HOW != kFftLanes && t < cols * q8; t += blockDim.x) {
      const int c = t / q8, j = t - c * q8;
      const double2 *xr = x + c * M + j;
      double2 *yr = y + c * M + 8 * j;
      const bool none = INT && zeros(xr[0].x, xr[0].y);  // see radix4's call
      if (none || radix8<INT>(f, xr, yr, q8, c8, inverse)) radix8<false>(f, xr, yr, q8, c8, inverse);
    }
    __syncthreads();
    double2 *tmp = x;
    x = y;
    y = tmp;
    Ns = 8;
  }
  const int q4 = M >> 2;
  for (; Ns < M; Ns <<= 2) {
    const int step = M / (4 * Ns);
    for (int t = threadIdx.x; HOW == kFftLanes && t < ((8 * cols * q4 + 31) & ~31); t += blockDim.x) {
      const bool in = t < 8 * cols * q4;
      const int b = in ? t >> 3 : 0, c = b / q4, j = b - c * q4, kk = j & (Ns - 1);
      const double2 *xr = x + c * M + j;
      double2 *yr = y + c * M + ((j - kk) << 2) + kk;
      if (Ns > 1)
        radix4_lanes<true>(f, xr, yr, q4, Ns, wm, kk * step, two, inverse, t & 7, in);
      else
        radix4_lanes<false>(f, xr, yr, q4, Ns, wm, 0, two, inverse, t & 7, in);
    }
    for (int t = threadIdx.x; HOW != kFftLanes && t < cols * q4; t += blockDim.x) {
      const int c = t / q4, j = t - c * q4;
      const int kk = j & (Ns - 1);
      const double2 *xr = x + c * M + j;
      double2 *yr = y + c * M + ((j - kk) << 2) + kk;
      // zeros (fluid at rest), which the integer forms would give up on: the first input tells
      const bool none = INT && zeros(xr[0].x, xr[0].y);
      if (Ns > 1) {
        if (none || radix4<INT, true>(f, xr, yr, q4, Ns, wm, kk * step, two, inverse))
          radix4<false, true>(f, xr, yr, q4, Ns, wm, kk * step, two, inverse);
      } else {
        if (none || radix4<INT, false>(f, xr, yr, q4, Ns, wm, 0, two, inverse))
          radix4<false, false>(f, xr, yr, q4, Ns, wm, 0, two, inverse);
      }
    }
    __syncthreads();
    double2 *tmp = x;
    x = y;
    y = tmp;
  }
  return x;
}

// Q: the right-hand side from the predictor's face values q = pd u* + pa e
// grad psi_old (ux, uy are qx, qy; egx, egy unused): 3 FP64 operations per
// cell instead of 7
template <int W, bool Q, int HOW>
__global__ void __launch_bounds__(256, HOW == kFftInt ? 4 : (HOW == kFftShort ? 5 : 1))
    k_poisson_fwd(Grid g, const double *__restrict__ sc, int k, const double *__restrict__ ux,
                  const double *__restrict__ uy, const double *__restrict__ egx, const double *__restrict__ egy,
                  const double2 *__restrict__ tw, double2 *__restrict__ spec) {
  pdl_entry();
  sc += (size_t)blockIdx.z * (kScalars);
  spec += (size_t)blockIdx.z * (g.css);
  extern __shared__ double2 smem[];
  const int ny = g.ny, M = ny >> 1;
  double2 *A = smem, *B = smem + W * M;
  double *Ad = reinterpret_cast<double *>(A);
  const int I0 = blockIdx.x * W + 1;
  const Fp64 f(blockIdx.x + threadIdx.x);
  const double pdx = sc[sc_pdx(k)], pdy = sc[sc_pdy(k)];
  for (int t = threadIdx.x; t < W * ny; t += blockDim.x) {
    const int c = t % W, r = t / W;
    const int I = I0 + c;
    double val = 0.;
    if (I <= g.nx) {
      // global rows of this case (the case's rows follow each other)
      const int zr = blockIdx.z * ny;
      const int rg = r + zr, rp = (r == ny - 1 ? 0 : r + 1) + zr;
      // differences of pax e grad psi_old and pay e grad psi_old across the
      // cell (its faces' values written by k_predict_mf or k_face_factor)
      if (Q) {
        val = f.add(f.sub(ux[ix(g, rg, I)], ux[ix(g, rg, I - 1)]), f.sub(uy[ix(g, rp, I)], uy[ix(g, rg, I)]));
      } else {
        const double X = egx[ix(g, rg, I)] - egx[ix(g, rg, I - 1)];
        const double Y = egy[ix(g, rp, I)] - egy[ix(g, rg, I)];
        const double dux = ux[ix(g, rg, I)] - ux[ix(g, rg, I - 1)];
        const double duy = uy[ix(g, rp, I)] - uy[ix(g, rg, I)];
        val = fma(pdx, dux, fma(pdy, duy, X + Y));
      }
    }
    Ad[c * ny + r] = val;
  }
  __syncthreads();
  double2 *Z = fft_rows<W, HOW>(A, B, M, tw, false, f, min(W, g.nx + 1 - I0));
  // the packed transform z_m, m < M; k_poisson_tdm does the real-to-complex
  // split (there the FP64 pipe has room)
  const int M1 = M + 1;
  for (int t = threadIdx.x; t < W * M; t += blockDim.x) {
    const int c = t / M, mm = t - c * M;
    const int I = I0 + c;
    if (I > g.nx) continue;
    spec[(size_t)(I - 1) * M1 + mm] = Z[c * M + mm];
  }
}

template <int W, int HOW>
__global__ void __launch_bounds__(256, HOW == kFftInt ? 4 : (HOW == kFftShort ? 5 : 1))
    k_poisson_inv(Grid g, const double2 *__restrict__ tw, const double2 *__restrict__ spec, double *__restrict__ psi) {
  pdl_entry();
  spec += (size_t)blockIdx.z * (g.css);
  extern __shared__ double2 smem[];
  const int ny = g.ny, M = ny >> 1, M1 = M + 1;
  double2 *A = smem, *B = smem + W * M;
  const int I0 = blockIdx.x * W + 1;
  const Fp64 f(blockIdx.x + threadIdx.x);
  for (int t = threadIdx.x; t < W * M; t += blockDim.x) {
    const int c = t / M, mm = t - c * M;
    const int I = I0 + c;
    // the packed input of the inverse transform, complex-to-real split done
    // by k_poisson_tdm
    A[c * M + mm] = I <= g.nx ? spec[(size_t)(I - 1) * M1 + mm] : make_double2(0., 0.);
  }
  __syncthreads();
  const double2 *zr = fft_rows<W, HOW>(A, B, M, tw, true, f, min(W, g.nx + 1 - I0));
  const double *xd = reinterpret_cast<const double *>(zr);
  for (int t = threadIdx.x; t < W * ny; t += blockDim.x) {
    const int c = t % W, r = t / W;
    const int I = I0 + c;
    if (I > g.nx) continue;
    const double v = xd[c * ny + r];
    const int rg = r + (int)blockIdx.z * ny;
    psi[ix(g, rg, I)] = v;
    if (I == 1) psi[ix(g, rg, 0)] = v;
    if (I == g.nx) psi[ix(g, rg, g.nx + 1)] = v;
  }
}

// Split of the packed transform of a wavenumber pair (real-to-complex, times
// 2): X_p = E + w^p O and X_{M-p} = conj E + w^{M-p} conj O with E = z_p +
// conj z_{M-p} and O = -i (z_p - conj z_{M-p}) (the pair's E and O with the
// signs of their imaginary parts flipped), products in FMAs.  Returns whether
// an integer form gave up (INT: the four sums and differences).
template <bool INT>
__device__ __forceinline__ bool split_pair(const Fp64 &f, double2 zm, double2 zr, double2 wa, double2 wb, double2 &xa,
                                           double2 &xb) {
  Fp64Int<INT> n(f);
  double2 E, O;
  n.addsubs(zr.x, zm.x, E.x, O.y);
  n.addsubs(zm.y, zr.y, O.x, E.y);
  xa = make_double2(fma(wa.x, O.x, fma(-wa.y, O.y, E.x)), fma(wa.x, O.y, fma(wa.y, O.x, E.y)));
  xb = make_double2(fma(wb.x, O.x, fma(wb.y, O.y, E.x)), fma(wb.y, O.x, fma(-wb.x, O.y, -E.y)));
  return INT && n.bad != 0;
}

// The way back, into the packed input of the inverse transform: z_p = E + i D
// conj w^p and z_{M-p} = conj E - i conj D conj w^{M-p}, with E = X_p + conj
// X_{M-p}, D = X_p - conj X_{M-p}; products in FMAs
template <bool INT>
__device__ __forceinline__ bool merge_pair(const Fp64 &f, double2 Xa, double2 Xb, double2 wa, double2 wb, double2 &za,
                                           double2 &zb) {
  Fp64Int<INT> n(f);
  double2 E, D;
  n.addsubs(Xa.x, Xb.x, E.x, D.x);
  n.addsubs(Xa.y, Xb.y, D.y, E.y);
  za = make_double2(fma(D.x, wa.y, fma(-D.y, wa.x, E.x)), fma(D.y, wa.y, fma(D.x, wa.x, E.y)));
  zb = make_double2(fma(-D.y, wb.x, fma(-D.x, wb.y, E.x)), fma(D.y, wb.y, fma(-D.x, wb.x, -E.y)));
  return INT && n.bad != 0;
}

// One lane's chunk of a system, rows x[0 .. L), factors f[k lanes].  AHEAD:
// the factors of the next kAhead rows are loaded while those of the present
// ones are used, since a block's shared memory leaves room for one to three
// warps a scheduler on large grids, which otherwise wait for them; what is
// left after the last whole group goes row by row (a test per row in every
// group, as a first version had it, takes an FP64 slot for each row past the
// end: 1300 x 1024, 21 rows a lane, 50 -> 42 us).  One launch of
// k_poisson_tdm, with the split's sums on the integer pipes: 2048 x 1024
// 61.7 -> 53 us, 4096 x 2048 472 -> 320 us (one warp a scheduler; four rows of
// the split's loads in flight as well).
constexpr int kAhead = 8;
template <bool AHEAD, int STEP, class Load, class Use>
__device__ __forceinline__ void sweep(int L, Load load, Use use) {
  auto row = [L](int k) { return STEP > 0 ? k : L - 1 - k; };
  if (!AHEAD) {
#pragma unroll 8
    for (int k = 0; k < L; ++k) use(row(k), load(row(k)));
    return;
  }
  decltype(load(0)) c[kAhead], n[kAhead];
  int k0 = 0;
  if (L >= kAhead) {
#pragma unroll
    for (int u = 0; u < kAhead; ++u) c[u] = load(row(u));
    for (; k0 + 2 * kAhead <= L; k0 += kAhead) {
#pragma unroll
      for (int u = 0; u < kAhead; ++u) n[u] = load(row(k0 + kAhead + u));
#pragma unroll
      for (int u = 0; u < kAhead; ++u) use(row(k0 + u), c[u]);
#pragma unroll
      for (int u = 0; u < kAhead; ++u) c[u] = n[u];
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u) use(row(k0 + u), c[u]);
    k0 += kAhead;
  }
#pragma unroll 4  // the step of 600 x 512, five rows a lane, 295.6 us; one row at a time 299.2
  for (; k0 < L; ++k0) use(row(k0), load(row(k0)));
}
// HOW a launch solves its chunks (chosen in tdm_how): plainly; chunks of up to
// kTdmReg rows in registers; shared with the integer pipes, factors ahead.
// Chunk<HOW> holds a lane's rows and factors between the sweeps.  In registers
// the factors load before the split's rows arrive: three trips to L2 and
// back, and the rows' to shared memory, leave the chain (k_poisson_tdm on
// 256 x 128 11.8 -> 9.0 us with the pairs' clusters at two
// warps a system, on 509 x 256 14.0 -> 11.4 us).
enum TdmHow { kTdmPlain, kTdmReg, kTdmInt };
constexpr int kTdmRegRows = 4;
template <int HOW>
struct Chunk {
  static constexpr bool INT = HOW == kTdmInt, reg = HOW == kTdmReg;
  static constexpr int kReg = reg ? kTdmRegRows : 1;
  const Fp64 &f64;
  const double4_32a *__restrict__ f;
  size_t lanes;
  int L;
  double *x;
  double4_32a c[kReg];
  double r[kReg];
  __device__ __forceinline__ Chunk(const Fp64 &f_, const double4_32a *fac, size_t lanes_, int L_, double *x_, bool act)
      : f64(f_), f(fac), lanes(lanes_), L(L_), x(x_) {
    if (reg && act) {
#pragma unroll
      for (int k = 0; k < kReg; ++k)
        if (k < L) c[k] = f[k * lanes];
    }
  }
  // forward from a zero carry, y_k = w_k r_k - v_k y_{k-1}; returns the last y
  __device__ __forceinline__ double forward() {
    double t = 0.;
    if (reg) {
#pragma unroll
      for (int k = 0; k < kReg; ++k)
        if (k < L) t = r[k] = fma(-c[k].y, t, f64.mul(c[k].x, x[k]));
      return t;
    }
    sweep<INT, 1>(
        L, [&](int k) { return make_double2(f[k * lanes].x, f[k * lanes].y); },
        [&](int k, double2 q) {
          t = fma(-q.y, t, f64.mul(q.x, x[k]));
          x[k] = t;
        });
    return t;
  }
  // the forward solution's fix-up by P_k carry and the backward sweep from a
  // zero carry, x_k = y_k - v_k x_{k+1}; returns the first x
  __device__ __forceinline__ double backward(double carry) {
    double u = 0.;
    if (reg) {
#pragma unroll
      for (int k = kReg - 1; k >= 0; --k)
        if (k < L) u = r[k] = fma(-c[k].y, u, fma(c[k].z, carry, r[k]));
      return u;
    }
    sweep<INT, -1>(
        L, [&](int k) { return make_double2(f[k * lanes].y, f[k * lanes].z); },
        [&](int k, double2 q) {
          u = fma(-q.x, u, fma(q.y, carry, x[k]));
          x[k] = u;
        });
    return u;
  }
  // the backward solution's fix-up by Q_k next
  __device__ __forceinline__ void fix(double next) {
    if (reg) {
#pragma unroll
      for (int k = 0; k < kReg; ++k)
        if (k < L) x[k] = fma(c[k].w, next, r[k]);
      return;
    }
    sweep<INT, 1>(
        L, [&](int k) { return f[k * lanes].w; }, [&](int k, double q) { x[k] = fma(q, next, x[k]); });
  }
  // P of the last row and Q of the first
  __device__ __forceinline__ double last_p() const {
    if (reg) {
      double v = c[0].z;
#pragma unroll
      for (int k = 1; k < kReg; ++k) v = k < L ? c[k].z : v;
      return v;
    }
    return f[(size_t)(L - 1) * lanes].z;
  }
  __device__ __forceinline__ double first_q() const { return reg ? c[0].w : f[0].w; }
};

// Tridiagonal solves along x, one per real system (y wavenumber m, real or
// imaginary part), one warp per system.  The pivots of the constant operator
// are precomputed, so the Thomas forward sweep is the first-order linear
// recurrence y_i = w_i r_i - v_i y_{i-1} and the back substitution is
// x_i = y_i - v_i x_{i+1}.  Lane l owns the L consecutive rows l*L..l*L+L-1:
// it runs both recurrences on its rows from a zero carry, the lanes combine
// their chunk maps (T, B): y -> T + B y with a shuffle scan, and each row is
// fixed up with the precomputed cumulative products P_i (forward) and Q_i
// (backward) of the recurrence coefficients inside its chunk.  Per row: 5
// FP64 operations instead of the 3 of a sequential sweep, but 32-way
// parallel per system.  fac[(m*L + k)*32 + l] = (w, v, P, Q) for row l*L+k.
// The singular m = 0 mode (Neumann in x, constant null space) has its last
// pivot pinned (w = v = 0) and is shifted to zero mean.
// Staging: per system a planar array with an odd lane stride S, in shared
// memory; when four systems of nx rows exceed it (nx above about 6900), in
// this block's slab of the global buffer stage (L2-resident, same arithmetic).
template <bool kGlobalStage, int HOW>
__global__ void __launch_bounds__(512)
    k_poisson_tdm(Grid g, int PB, int G, int L, int S, const double4_32a *__restrict__ fac,
                  const double2 *__restrict__ tw, double2 *__restrict__ spec, double *__restrict__ stage) {
  pdl_entry();
  extern __shared__ double2 smem_d2[];
  __shared__ double xch[16][4][2];  // per system of the block, per warp of the system: a chunk-map total
  const Fp64 f64(blockIdx.x + threadIdx.x);
  const int nx = g.nx, M = g.ny / 2, M1 = M + 1;
  const int p0 = blockIdx.x * PB;
  const int np = min(PB, M / 2 + 1 - p0);  // pairs (p, M - p), p = 0 .. M/2
  const int lanes = 32 * G;                // chunks per system
  const int sys_len = lanes * S;
  double *sm = kGlobalStage ? stage + ((size_t)blockIdx.z * gridDim.x + blockIdx.x) * 4 * PB * sys_len
                            : reinterpret_cast<double *>(smem_d2);
  double2 *sp = spec + (size_t)blockIdx.z * g.css;
  // warp -> system (4 per pair) and its part sub of G; chunk j of the
  // system = this lane's L rows
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sys = warp / G, sub = warp - sys * G, j = sub * 32 + lane;
  const bool act = sys < 4 * np;  // warp-uniform
  const int pq = p0 + (sys >> 2);
  const int m = (sys & 2) ? M - pq : pq;  // the wavenumber of this system
  double *x = sm + sys * sys_len + j * S;
  const double4_32a *f = fac + (size_t)m * L * lanes + j;
  constexpr bool INT = HOW == kTdmInt;
  Chunk<HOW> ch(f64, f, lanes, L, x, act);
  // ---- load the packed transform of both wavenumbers of each pair, split
  // it (real-to-complex, times 2: X_m = (z_m + conj z_{M-m}) + w^m (-i)(z_m -
  // conj z_{M-m})) into four planar systems: X_p re, im, X_{M-p} re, im
  // (kBatch rows' loads in flight: the stores to sm keep the compiler from
  // moving the next rows' loads above them)
  constexpr int kBatch = INT ? 4 : 1;
  const int rows = lanes * L * np;
  for (int t0 = threadIdx.x; t0 < rows; t0 += kBatch * blockDim.x) {
    double2 zm[kBatch], zr[kBatch];
#pragma unroll
    for (int v = 0; v < kBatch; ++v) {
      const int t = t0 + v * blockDim.x, i = t / np, p = p0 + (t - i * np);
      if (t < rows && i < nx) {
        zm[v] = sp[(size_t)i * M1 + p];
        zr[v] = sp[(size_t)i * M1 + (p == 0 ? 0 : M - p)];
      }
    }
#pragma unroll
    for (int v = 0; v < kBatch; ++v) {
      const int t = t0 + v * blockDim.x, i = t / np, q = t - i * np, p = p0 + q;
      if (t >= rows) break;
      double2 xa = make_double2(0., 0.), xb = make_double2(0., 0.);
      if (i < nx) {
        const double2 wa = tw[p], wb = tw[M - p];
        const bool none = INT && zeros(zm[v].x, zm[v].y, zr[v].x, zr[v].y);
        if (none || split_pair<INT>(f64, zm[v], zr[v], wa, wb, xa, xb)) split_pair<false>(f64, zm[v], zr[v], wa, wb, xa, xb);
      }
      double *o = sm + (size_t)(4 * q) * sys_len + (i / L) * S + (i % L);
      o[0] = xa.x;
      o[sys_len] = xa.y;
      o[2 * sys_len] = xb.x;
      o[3 * sys_len] = xb.y;
    }
  }
  __syncthreads();
  double T = 0., B = 0.;
  if (act) {
    // forward, local from a zero carry
    T = ch.forward();
    B = ch.last_p();
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const double Tp = __shfl_up_sync(0xffffffffu, T, d), Bp = __shfl_up_sync(0xffffffffu, B, d);
      if (lane >= d) {
        T = fma(B, Tp, T);
        B = f64.mul(B, Bp);
      }
    }
  }
  // the map of the system's chunks before this warp's (G > 1: warp totals)
  double Cin = 0.;
  if (G > 1) {
    if (act && lane == 31) {
      xch[sys][sub][0] = T;
      xch[sys][sub][1] = B;
    }
    __syncthreads();
    if (act)
      for (int q = 0; q < sub; ++q) Cin = fma(xch[sys][q][1], Cin, xch[sys][q][0]);
    __syncthreads();
  }
  double Sx = 0., Cc = 0.;
  if (act) {
    const double Tu = __shfl_up_sync(0xffffffffu, T, 1), Bu = __shfl_up_sync(0xffffffffu, B, 1);
    const double carry = lane == 0 ? Cin : fma(Bu, Cin, Tu);
    // fix up the forward solution, then the backward sweep from a zero carry
    Sx = ch.backward(carry);
    Cc = ch.first_q();
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const double Sp = __shfl_down_sync(0xffffffffu, Sx, d), Cp = __shfl_down_sync(0xffffffffu, Cc, d);
      if (lane + d < 32) {
        Sx = fma(Cc, Sp, Sx);
        Cc = f64.mul(Cc, Cp);
      }
    }
  }
  // the map of the chunks after this warp's
  double Din = 0.;
  if (G > 1) {
    if (act && lane == 0) {
      xch[sys][sub][0] = Sx;
      xch[sys][sub][1] = Cc;
    }
    __syncthreads();
    if (act)
      for (int q = G - 1; q > sub; --q) Din = fma(xch[sys][q][1], Din, xch[sys][q][0]);
    __syncthreads();
  }
  // the singular mode m = 0 (systems 0, 1 of pair 0): zero mean over x, imaginary part 0
  const bool gauge = act && m == 0 && (sys & 2) == 0;
  double acc = 0.;
  if (act) {
    const double Sd = __shfl_down_sync(0xffffffffu, Sx, 1), Cd = __shfl_down_sync(0xffffffffu, Cc, 1);
    const double next = lane == 31 ? Din : fma(Cd, Din, Sd);
    ch.fix(next);
    if (gauge) {
      for (int k = 0; k < L; ++k) acc += (j * L + k < nx) ? x[k] : 0.;
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
    }
  }
  if (G > 1) {
    if (gauge && lane == 0) xch[sys][sub][0] = acc;
    __syncthreads();
    if (gauge) {
      acc = 0.;
      for (int q = 0; q < G; ++q) acc += xch[sys][q][0];
    }
  }
  if (gauge) {
    const double mean = (sys & 1) ? 0. : acc / nx;
    for (int k = 0; k < L; ++k) x[k] = (sys & 1) ? 0. : x[k] - mean;
  }
  __syncthreads();
  // ---- complex-to-real split of the solved pair into the packed input of the
  // inverse transform: z_m = E + i O, E = X_m + conj X_{M-m},
  // O = (X_m - conj X_{M-m}) conj w^m, for m = p and m = M - p (< M)
  for (int t = threadIdx.x; t < nx * np; t += blockDim.x) {
    const int i = t / np, q = t - i * np;
    const int p = p0 + q;
    const int at = (i / L) * S + (i % L);
    const double2 Xa = make_double2(sm[(4 * q) * sys_len + at], sm[(4 * q + 1) * sys_len + at]);
    const double2 Xb = make_double2(sm[(4 * q + 2) * sys_len + at], sm[(4 * q + 3) * sys_len + at]);
    const double2 wa = tw[p], wb = tw[M - p];
    double2 za, zb;
    const bool none = INT && zeros(Xa.x, Xa.y, Xb.x, Xb.y);
    if (none || merge_pair<INT>(f64, Xa, Xb, wa, wb, za, zb)) merge_pair<false>(f64, Xa, Xb, wa, wb, za, zb);
    sp[(size_t)i * M1 + p] = za;
    if (p != 0 && 2 * p != M) sp[(size_t)i * M1 + (M - p)] = zb;
  }
}

// The same solves with CL = 2 or 4 warps per system, spread over a cluster of
// CL CTAs: CTA r of a cluster owns rows 32 L r .. 32 L (r + 1) - 1 of the four
// systems of one wavenumber pair (warp s: system s), so a launch has CL CTAs
// per pair where k_poisson_tdm has one block per pair or two, and the CL
// (ny/4 + 1) CTAs of a case even out over the SMs (in a launch of blocks of
// one or two pairs, ny/4 + 1 pairs leave SMs idle while the last blocks run,
// one in six for ny = 1024).  The chunk-map totals of the other CTAs come
// through distributed shared memory and are combined in the order
// k_poisson_tdm<false> combines its warps' at G = CL, so both give the same
// bits.  L = tdm_chunk(nx, CL), S = L | 1; fac is the G = CL table.
template <int HOW, int CL>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(128)
    k_poisson_tdm_cl(Grid g, int L, int S, const double4_32a *__restrict__ fac, const double2 *__restrict__ tw,
                     double2 *__restrict__ spec) {
  pdl_entry();
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  extern __shared__ double smem_cl[];
  // per system: forward (T, B) and backward (S, C) totals of this CTA's warp, the gauge sum
  __shared__ double xf[4][2], xb[4][2], xg[4];
  const Fp64 f64(blockIdx.x + threadIdx.x);
  const int nx = g.nx, M = g.ny / 2, M1 = M + 1;
  const int rank = (int)cl.block_rank();
  const int p = (int)blockIdx.x / CL;  // the pair (p, M - p), p = 0 .. M/2
  const int rows = 32 * L, r0 = rank * rows;   // this CTA's rows r0 .. r0 + rows - 1
  const int sys_len = 32 * S;
  double2 *sp = spec + (size_t)blockIdx.z * g.css;
  const int sys = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int lanes = 32 * CL, j = rank * 32 + lane;  // chunk of the system
  const int m = (sys & 2) ? M - p : p;
  double *x = smem_cl + sys * sys_len + lane * S;
  const double4_32a *f = fac + (size_t)m * L * lanes + j;
  constexpr bool INT = HOW == kTdmInt;
  Chunk<HOW> ch(f64, f, lanes, L, x, true);
  // ---- load and split (as in k_poisson_tdm), this CTA's rows
  for (int t = threadIdx.x; t < rows; t += blockDim.x) {
    const int i = r0 + t;
    const int at = (t / L) * S + (t % L);
    double2 xa = make_double2(0., 0.), xbv = make_double2(0., 0.);
    if (i < nx) {
      const double2 zm = sp[(size_t)i * M1 + p];
      const double2 zr = sp[(size_t)i * M1 + (p == 0 ? 0 : M - p)];
      const double2 wa = tw[p], wb = tw[M - p];
      const bool none = INT && zeros(zm.x, zm.y, zr.x, zr.y);
      if (none || split_pair<INT>(f64, zm, zr, wa, wb, xa, xbv)) split_pair<false>(f64, zm, zr, wa, wb, xa, xbv);
    }
    smem_cl[0 * sys_len + at] = xa.x;
    smem_cl[1 * sys_len + at] = xa.y;
    smem_cl[2 * sys_len + at] = xbv.x;
    smem_cl[3 * sys_len + at] = xbv.y;
  }
  __syncthreads();
  double T, B;
  {
    T = ch.forward();
    B = ch.last_p();
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const double Tp = __shfl_up_sync(0xffffffffu, T, d), Bp = __shfl_up_sync(0xffffffffu, B, d);
      if (lane >= d) {
        T = fma(B, Tp, T);
        B = f64.mul(B, Bp);
      }
    }
  }
  if (lane == 31) {
    xf[sys][0] = T;
    xf[sys][1] = B;
  }
  cl.sync();
  double Cin = 0.;
  for (int q = 0; q < rank; ++q) {
    const double *o = cl.map_shared_rank(&xf[sys][0], q);
    Cin = fma(o[1], Cin, o[0]);
  }
  double Sx, Cc;
  {
    const double Tu = __shfl_up_sync(0xffffffffu, T, 1), Bu = __shfl_up_sync(0xffffffffu, B, 1);
    const double carry = lane == 0 ? Cin : fma(Bu, Cin, Tu);
    Sx = ch.backward(carry);
    Cc = ch.first_q();
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const double Sp = __shfl_down_sync(0xffffffffu, Sx, d), Cp = __shfl_down_sync(0xffffffffu, Cc, d);
      if (lane + d < 32) {
        Sx = fma(Cc, Sp, Sx);
        Cc = f64.mul(Cc, Cp);
      }
    }
  }
  if (lane == 0) {
    xb[sys][0] = Sx;
    xb[sys][1] = Cc;
  }
  cl.sync();
  double Din = 0.;
  for (int q = CL - 1; q > rank; --q) {
    const double *o = cl.map_shared_rank(&xb[sys][0], q);
    Din = fma(o[1], Din, o[0]);
  }
  {
    const double Sd = __shfl_down_sync(0xffffffffu, Sx, 1), Cd = __shfl_down_sync(0xffffffffu, Cc, 1);
    const double next = lane == 31 ? Din : fma(Cd, Din, Sd);
    ch.fix(next);
  }
  // the singular mode m = 0 (systems 0, 1 of pair 0): zero mean over x,
  // imaginary part 0 (p is the same on the whole cluster)
  if (p == 0) {
    const bool gauge = (sys & 2) == 0;
    double acc = 0.;
    if (gauge) {
      for (int k = 0; k < L; ++k) acc += (j * L + k < nx) ? x[k] : 0.;
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
      if (lane == 0) xg[sys] = acc;
    }
    cl.sync();
    if (gauge) {
      acc = 0.;
      for (int q = 0; q < CL; ++q) acc += *cl.map_shared_rank(&xg[sys], q);
      const double mean = (sys & 1) ? 0. : acc / nx;
      for (int k = 0; k < L; ++k) x[k] = (sys & 1) ? 0. : x[k] - mean;
    }
  }
  // no CTA of the cluster reads another's shared memory after this point
  cl.sync();
  // ---- complex-to-real split (as in k_poisson_tdm), this CTA's rows
  for (int t = threadIdx.x; t < rows; t += blockDim.x) {
    const int i = r0 + t;
    if (i >= nx) break;
    const int at = (t / L) * S + (t % L);
    const double2 Xa = make_double2(smem_cl[0 * sys_len + at], smem_cl[1 * sys_len + at]);
    const double2 Xb = make_double2(smem_cl[2 * sys_len + at], smem_cl[3 * sys_len + at]);
    const double2 wa = tw[p], wb = tw[M - p];
    double2 za, zb;
    const bool none = INT && zeros(Xa.x, Xa.y, Xb.x, Xb.y);
    if (none || merge_pair<INT>(f64, Xa, Xb, wa, wb, za, zb)) merge_pair<false>(f64, Xa, Xb, wa, wb, za, zb);
    sp[(size_t)i * M1 + p] = za;
    if (p != 0 && 2 * p != M) sp[(size_t)i * M1 + (M - p)] = zb;
  }
}

// ---------------------------------------------------------------------------
// velocity correction (+ pressure update)
//   src/fluid/correct_velocity/ux.c:18-66, uy.c:17-64
//   src/fluid/update_pressure.c:7-53
//   u -= dt_new / rho_ref dpsi_new / h;  u += -dt_old (1/rho - 1/rho_ref) dpsi_old / h
//   with 1/rho - 1/rho_ref = e / rho_ref; pax e dpsi_old and pay e dpsi_old at
//   the faces are egx, egy (k_predict_mf or k_face_factor); the x coefficients
//   come per column (cnew / HXXF(I), cold / HXXF(I) / pax), the y ones per case
// thread (I, J): I = 1..nx
// ---------------------------------------------------------------------------
// DP: also stores psi_new's differences across the faces for the next
// substage's predictor (dpx, dpy; the fused step)
template <bool PRES, bool DP>
__global__ void __launch_bounds__(BX *BY)
    k_correct(Grid g, const double *__restrict__ sc, const double *__restrict__ coltab, int k,
              double *__restrict__ ux, double *__restrict__ uy, const double *__restrict__ psin,
              const double *__restrict__ egx, const double *__restrict__ egy, double *__restrict__ p,
              double *__restrict__ dpx, double *__restrict__ dpy) {
  pdl_entry();
  sc += (size_t)blockIdx.z * (kScalars);
  const double *__restrict__ ct = coltab + (size_t)blockIdx.z * 3 * kColTabs * g.ct;
  const double *__restrict__ cn = ct + ct_cnewx(k) * g.ct, *__restrict__ co = ct + ct_coldx(k) * g.ct;
  const int I = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int J = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (I > g.nx || J > g.ny) return;
  const int zr = blockIdx.z * g.ny;  // first row of this case
  const int r = J - 1 + zr, rm = wrap(J - 1, g.ny) + zr;
  const double cnewy = sc[sc_cnewy(k)], coldyp = sc[sc_coldyp(k)];
  const Fp64 f(I);
  const double pn0 = psin[ix(g, r, I)];
  if (I >= 2) {
    double u = ux[ix(g, r, I - 1)];
    const double d = f.sub(pn0, psin[ix(g, r, I - 1)]);
    if (DP) dpx[ix(g, r, I - 1)] = d;
    u = fma(-cn[I], d, u);
    u = fma(co[I], egx[ix(g, r, I - 1)], u);
    ux[ix(g, r, I - 1)] = u;
  }
  {
    double u = uy[ix(g, r, I)];
    const double d = f.sub(pn0, psin[ix(g, rm, I)]);
    if (DP) dpy[ix(g, r, I)] = d;
    u = fma(-cnewy, d, u);
    u = fma(coldyp, egy[ix(g, r, I)], u);
    uy[ix(g, r, I)] = u;
  }
  if (I == 1) {
    ux[ix(g, r, 0)] = 0.;
    uy[ix(g, r, 0)] = 0.;
  }
  if (I == g.nx) {
    ux[ix(g, r, g.nx)] = 0.;
    uy[ix(g, r, g.nx + 1)] = 0.;
  }
  if (PRES) {
    const double pv = f.add(p[ix(g, r, I)], pn0);
    p[ix(g, r, I)] = pv;
    if (I == 1) p[ix(g, r, 0)] = pv;
    if (I == g.nx) p[ix(g, r, g.nx + 1)] = pv;
  }
}

// pressure update alone (fine-grained entry point); I = 1..nx
__global__ void k_pressure(Grid g, const double *__restrict__ psin, double *__restrict__ p) {
  pdl_entry();
  const int I = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int J = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (I > g.nx || J > g.ny) return;
  const int r = J - 1;
  const double pv = p[ix(g, r, I)] + psin[ix(g, r, I)];
  p[ix(g, r, I)] = pv;
  if (I == 1) p[ix(g, r, 0)] = pv;
  if (I == g.nx) p[ix(g, r, g.nx + 1)] = pv;
}

// ---------------------------------------------------------------------------
// time step size (src/decide_dt.c:34-169)
// min over faces of h / (|u| + 1e-8) equals h / (max |u| + 1e-8) for a
// fixed h because both roundings are monotone; so k_decide_dt reduces max |u|
// per x column (ux) and over the domain (uy) on the integer patterns of the
// non-negative doubles, and k_decide_dt_fin forms the nx - 1 quotients of the
// columns over its blocks and their minimum (the minimum of positive doubles
// is that of their bit patterns), then its last block the dt and every
// per-substage scalar of the step.  A non-finite velocity sets bit 0 of the
// status word.  Scratch per case (nx + 8 words, zero between launches):
// [2..nx] column max |ux| bits, [nx+2] max |uy| bits, [nx+4] the complement
// of the least quotient's bits (so that zero means none yet), [nx+5] the
// finishing blocks' counter, [nx+6] whether any ux is not zero.
// ---------------------------------------------------------------------------
constexpr unsigned long long kAbsMask = 0x7fffffffffffffffULL;
constexpr unsigned long long kInfBits = 0x7ff0000000000000ULL;

__global__ void __launch_bounds__(BX *BY)
    k_decide_dt(Grid g, const double *__restrict__ ux, const double *__restrict__ uy,
                unsigned long long *__restrict__ acc) {
  pdl_entry();
  acc += (size_t)blockIdx.z * ((size_t)g.nx + 8);
  __shared__ unsigned long long colmax[BY][BX];
  __shared__ unsigned long long ymax[BY * BX];
  const int I = blockIdx.x * BX + threadIdx.x + 1;  // 1..nx+1
  unsigned long long mx = 0ULL, my = 0ULL;
  if (I <= g.nx) {
#pragma unroll 4
    for (int J = blockIdx.y * BY + threadIdx.y + 1; J <= g.ny; J += gridDim.y * BY) {
      const int r = J - 1 + (int)blockIdx.z * g.ny;
      if (I >= 2) {
        const unsigned long long b = (unsigned long long)dbits(ux[ix(g, r, I - 1)]) & kAbsMask;
        mx = b > mx ? b : mx;
      }
      const unsigned long long c = (unsigned long long)dbits(uy[ix(g, r, I)]) & kAbsMask;
      my = c > my ? c : my;
    }
  }
  colmax[threadIdx.y][threadIdx.x] = mx;
  const int tid = threadIdx.y * BX + threadIdx.x;
  ymax[tid] = my;
  __syncthreads();
  if (threadIdx.y == 0) {
    unsigned long long v = 0ULL;
    for (int k = 0; k < BY; ++k) v = colmax[k][threadIdx.x] > v ? colmax[k][threadIdx.x] : v;
    if (I <= g.nx && v) atomicMax(acc + I, v);
  }
  for (int w = BX * BY / 2; w > 0; w >>= 1) {
    if (tid < w) ymax[tid] = ymax[tid + w] > ymax[tid] ? ymax[tid + w] : ymax[tid];
    __syncthreads();
  }
  if (tid == 0 && ymax[0]) atomicMax(acc + g.nx + 2, ymax[0]);
}

// the finishing kernel: one column per thread (I = 2..nx over the blocks),
// then the last block of each case: dt, the scalars and the reset of the
// scratch
constexpr int kDtFinThreads = 256;
__global__ void __launch_bounds__(kDtFinThreads)
    k_decide_dt_fin(Grid g, Metrics m, Phys ph0, unsigned long long *__restrict__ acc, double *__restrict__ sc,
                    int *__restrict__ status, double dt_fixed, double coef_adv) {
  pdl_entry();
  const Phys ph = zphys(g, ph0);
  if (g.phys) dt_fixed = ph.dtfix;
  acc += (size_t)blockIdx.z * ((size_t)g.nx + 8);
  sc += (size_t)blockIdx.z * (kScalars);
  status += (size_t)blockIdx.z * (1);
  __shared__ double wmin[kDtFinThreads / 32];
  __shared__ int wbad[kDtFinThreads / 32];
  __shared__ bool last;
  __shared__ double dt_sh;
  __shared__ int flow_sh;
  const double small = 1.e-8;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // dt_adv = coef * min(1, min_i hx_i / (max|ux|_i + small), hy / (max|uy| + small))
  double d = 1.;
  int bad = 0;
  const int i = blockIdx.x * kDtFinThreads + tid + 2;  // column i, and nx + 1 for the uy quotient
  if (i <= g.nx + 1) {
    // the maxima are final (the stream order) and were formed at L2
    const unsigned long long b = __ldcg(acc + (i <= g.nx ? i : g.nx + 2));
    bad = (b >= kInfBits ? 1 : 0) | (b != 0 && i <= g.nx ? 2 : 0);  // bit 1: there is flow along x
    d = (i <= g.nx ? m.hxxf[i] : g.hy) / (__longlong_as_double((long long)b) + small);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    d = fmin(d, __shfl_xor_sync(0xffffffffu, d, o));
    bad |= __shfl_xor_sync(0xffffffffu, bad, o);
  }
  if (lane == 0) {
    wmin[warp] = d;
    wbad[warp] = bad;
  }
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < kDtFinThreads / 32; ++w) {
      d = fmin(d, wmin[w]);
      bad |= wbad[w];
    }
    if (bad & 1) atomicOr(status, 1);
    last = true;
    if (gridDim.x > 1) {
      if (bad & 2) atomicOr(acc + g.nx + 6, 1ULL);
      // a positive d (or 1): the least bit pattern is the least value
      atomicMax(acc + g.nx + 4, ~(unsigned long long)dbits(d));
      __threadfence();
      const unsigned int done = atomicAdd(reinterpret_cast<unsigned int *>(acc + g.nx + 5), 1u);
      last = (done == gridDim.x - 1);
    }
    dt_sh = d;
    flow_sh = bad & 2;
  }
  __syncthreads();
  if (!last) return;
  // per-substage scalars; RK3 coefficients of src/runge_kutta.c:8-15.  Lane k
  // < 3 takes substage k, lane k + 3 its dtold / dtnew beside lane k's refden
  // / dtnew (an FP64 instruction takes the warp's slot once for all of them)
  if (warp == 0) {
    double dt = dt_sh;
    bool flow = flow_sh != 0;
    if (gridDim.x > 1) {
      __threadfence();
      flow = __ldcg(acc + g.nx + 6) != 0;
      dt = __longlong_as_double((long long)~__ldcg(acc + g.nx + 4));
    }
    // the 1 of the minimum stands here: with nx a multiple of kDtFinThreads
    // every thread above has a quotient in its place
    // (by words: any positive value above 1, and any NaN)
    if ((unsigned long long)dbits(dt) > (unsigned long long)dbits(1.)) dt = 1.;
    dt *= coef_adv;
    dt = fmin(dt, dt_fixed);
    const int k = lane % 3, ko = (k + 2) % 3;
    const double al[3] = {32. / 60., 25. / 60., 45. / 60.};
    const double be[3] = {0. / 60., -17. / 60., -25. / 60.};
    const double abo = ko == 0 ? al[0] + be[0] : (ko == 1 ? al[1] + be[1] : al[2] + be[2]);
    const double ab = k == 0 ? al[0] + be[0] : (k == 1 ? al[1] + be[1] : al[2] + be[2]);
    const double a = k == 0 ? al[0] : (k == 1 ? al[1] : al[2]), b = k == 0 ? be[0] : (k == 1 ? be[1] : be[2]);
    const double dtold = abo * dt, dtnew = ab * dt;
    const double quo = (lane < 3 ? ph.refden : dtold) / dtnew;
    const double ratio = __shfl_down_sync(0xffffffffu, quo, 3);
    if (lane < 3) {
      const double gdt2 = 2. * dtnew;
      const double cdiv = quo * (0.5 / g.ny);
      const double cadd = -ratio * (0.5 / g.ny);
      const double pax = cadd * (g.idx * g.idx), pay = cadd * (g.ihy * g.ihy);
      const double cnew = dtnew * ph.irefden, cold = -dtold * ph.irefden, coldy = cold * g.ihy;
      if (k == 0) {
        sc[0] = dt;
        sc[kScStill] = flow ? 0. : 1.;
      }
      sc[sc_adt(k)] = a * dt;
      sc[sc_bdt(k)] = b * dt;
      sc[sc_gdt(k)] = dtnew;
      sc[sc_adt2(k)] = 2. * (a * dt);
      sc[sc_bdt2(k)] = 2. * (b * dt);
      sc[sc_gdt2(k)] = gdt2;
      sc[sc_dtold(k)] = dtold;
      sc[sc_dtnew(k)] = dtnew;
      sc[sc_pdx(k)] = cdiv * g.idx;
      sc[sc_pdy(k)] = cdiv * g.ihy;
      sc[sc_pax(k)] = pax;
      sc[sc_pay(k)] = pay;
      sc[sc_cnew(k)] = cnew;
      sc[sc_cold(k)] = cold;
      sc[sc_cnewy(k)] = cnew * g.ihy;
      sc[sc_coldy(k)] = coldy;
      sc[sc_gdt2y(k)] = gdt2 * g.ihy;
      sc[sc_coldyp(k)] = coldy / pay;
      sc[sc_rpx(k)] = ph.rref2 * pax;
      sc[sc_rpy(k)] = ph.rref2 * pay;
    }
  }
  __syncthreads();
  // reset the scratch for the next launch
  for (int t = tid; t <= g.nx + 6; t += kDtFinThreads) acc[t] = 0ULL;
}

// the per-column coefficients of the three substages from the scalars (one
// column per thread, over many blocks: on one block they were the finishing
// kernel's tail)
__global__ void __launch_bounds__(kDtFinThreads)
    k_decide_dt_tab(Grid g, Metrics m, const double *__restrict__ sc, double *__restrict__ coltab) {
  pdl_entry();
  sc += (size_t)blockIdx.z * (kScalars);
  coltab += (size_t)blockIdx.z * 3 * kColTabs * g.ct;
  const int I = blockIdx.x * kDtFinThreads + threadIdx.x;
  if (I > g.nx + 1) return;
  const double ih = m.ihxxf[I];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    // cold / pax once per column and substage (the same quotient everywhere)
    const double cop = sc[sc_cold(k)] / sc[sc_pax(k)];
    coltab[(size_t)ct_gdt2x(k) * g.ct + I] = sc[sc_gdt2(k)] * ih;
    coltab[(size_t)ct_cnewx(k) * g.ct + I] = sc[sc_cnew(k)] * ih;
    coltab[(size_t)ct_coldx(k) * g.ct + I] = cop * ih;
  }
}

// pax e grad psi_old and pay e grad psi_old, e = rho_ref / rho - 1, at ux
// faces (I = 1..nx+1) and uy faces (I = 1..nx) from a density field and
// psi_old, as k_predict_mf stores them (fine-grained entry points; the
// scalars of slot 0)
__global__ void k_face_factor(Grid g, const double *__restrict__ sc, const double *__restrict__ den,
                              const double *__restrict__ psio, double *__restrict__ egx, double *__restrict__ egy) {
  pdl_entry();
  const int I = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int J = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (I > g.nx + 1 || J > g.ny) return;
  const int r = J - 1, rm = wrap(J - 1, g.ny);
  const double ps = psio[ix(g, r, I)];
  const double ex = fma(sc[sc_rpx(0)], rcp_nr(den[ix(g, r, I - 1)] + den[ix(g, r, I)]), -sc[sc_pax(0)]);
  egx[ix(g, r, I - 1)] = ex * (ps - psio[ix(g, r, I - 1)]);
  if (I <= g.nx) {
    const double ey = fma(sc[sc_rpy(0)], rcp_nr(den[ix(g, rm, I)] + den[ix(g, r, I)]), -sc[sc_pay(0)]);
    egy[ix(g, r, I)] = ey * (ps - psio[ix(g, rm, I)]);
  }
}

// ---------------------------------------------------------------------------
// diagnostics of the reference's log files (src/logging/), reduced on the device:
//   [0] max |div u|                     src/logging/divergence.c:41-64
//   [1] min vof, [2] max vof, [3] sum vof J, [4] sum J, [5] interface area
//                                       src/logging/interface.c:34-65
//   [6..7] momentum x, y                src/logging/momentum.c:40-56
//   [8..9] kinetic energy x, y          src/logging/energy.c:42-58
//   [10..11] max |ux|, max |uy|         src/logging/extrema.c:25-38
//   [12..13] wall shear stress x = 0, lx  src/logging/stress.c:29-35
// Per-block partials in a fixed order, then one block: deterministic.
// ---------------------------------------------------------------------------
constexpr int kDiag = 16;

__device__ __forceinline__ void block_reduce(double (*sm)[BX * BY], int tid, const double *v) {
  for (int q = 0; q < kDiag; ++q) sm[q][tid] = v[q];
  __syncthreads();
  for (int w = BX * BY / 2; w > 0; w >>= 1) {
    if (tid < w) {
      for (int q = 0; q < kDiag; ++q) {
        const double a = sm[q][tid], b = sm[q][tid + w];
        // 0 and 2 and 10..11 are maxima, 1 is a minimum, the rest sums
        sm[q][tid] = (q == 0 || q == 2 || q == 10 || q == 11) ? fmax(a, b) : (q == 1 ? fmin(a, b) : a + b);
      }
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(BX *BY)
    k_diag_partial(Grid g, Metrics m, const double *__restrict__ ux, const double *__restrict__ uy,
                   const double *__restrict__ vof, const double *__restrict__ den, const double *__restrict__ txy,
                   double nu, double *__restrict__ part) {
  pdl_entry();
  __shared__ double sm[kDiag][BX * BY];
  const int I = blockIdx.x * BX + threadIdx.x + 1;
  const int J = blockIdx.y * BY + threadIdx.y + 1;
  const int tid = threadIdx.y * BX + threadIdx.x;
  double v[kDiag];
  for (int q = 0; q < kDiag; ++q) v[q] = 0.;
  v[1] = 1.;  // the reference starts min at 1 and max at 0
  if (I <= g.nx && J <= g.ny) {
    const int r = J - 1, rm = wrap(J - 1, g.ny), rp = wrap(J + 1, g.ny);
    const double jdxc = g.dx * g.hy;
    const double div = (ux[ix(g, r, I)] - ux[ix(g, r, I - 1)]) * g.idx + (uy[ix(g, rp, I)] - uy[ix(g, r, I)]) * g.ihy;
    v[0] = fabs(div);
    const double phi = vof[ix(g, r, I)];
    v[1] = phi;
    v[2] = phi;
    v[3] = phi * jdxc;
    v[4] = jdxc;
    v[5] = fabs(phi - vof[ix(g, r, I - 1)]) * g.hy + fabs(phi - vof[ix(g, rm, I)]) * g.dx;
    if (I == g.nx) v[5] += fabs(vof[ix(g, r, g.nx + 1)] - phi) * g.hy;
    if (I >= 2) {
      const double u = ux[ix(g, r, I - 1)];
      const double jdxf = m.hxxf[I] * g.hy;
      const double rho = 0.5 * den[ix(g, r, I - 1)] + 0.5 * den[ix(g, r, I)];
      v[6] = rho * u * jdxf;
      v[8] = 0.5 * rho * u * u * jdxf;
      v[10] = fabs(u);
    }
    const double w = uy[ix(g, r, I)];
    const double rhoy = 0.5 * den[ix(g, rm, I)] + 0.5 * den[ix(g, r, I)];
    v[7] = rhoy * w * jdxc;
    v[9] = 0.5 * rhoy * w * w * jdxc;
    v[11] = fabs(w);
    // JDXF / HXXF = hy at the wall faces
    if (I == 1) v[12] = nu * g.hy * txy[ix(g, r, 0)];
    if (I == g.nx) v[13] = nu * g.hy * txy[ix(g, r, g.nx)];
  }
  block_reduce(sm, tid, v);
  if (tid < kDiag) part[(size_t)(blockIdx.y * gridDim.x + blockIdx.x) * kDiag + tid] = sm[tid][0];
}

__global__ void __launch_bounds__(BX *BY) k_diag_final(const double *__restrict__ part, int nblocks,
                                                       double *__restrict__ out) {
  pdl_entry();
  __shared__ double sm[kDiag][BX * BY];
  const int tid = threadIdx.x;
  double v[kDiag];
  for (int q = 0; q < kDiag; ++q) v[q] = 0.;
  v[1] = 1.;
  for (int b = tid; b < nblocks; b += BX * BY) {
    for (int q = 0; q < kDiag; ++q) {
      const double x = part[(size_t)b * kDiag + q];
      v[q] = (q == 0 || q == 2 || q == 10 || q == 11) ? fmax(v[q], x) : (q == 1 ? fmin(v[q], x) : v[q] + x);
    }
  }
  block_reduce(sm, tid, v);
  if (tid < kDiag) out[tid] = sm[tid][0];
}

// running sums of the statistics (src/statistics.c:99-151): ux1 += ux over
// I = 1..nx+1, uy1 += uy and vof1 += vof over I = 0..nx+1
__global__ void k_stats_collect(Grid g, const double *__restrict__ ux, const double *__restrict__ uy,
                                const double *__restrict__ vof, double *__restrict__ ux1, double *__restrict__ uy1,
                                double *__restrict__ vof1) {
  pdl_entry();
  const int I = blockIdx.x * blockDim.x + threadIdx.x;
  const int J = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (I > g.nx + 1 || J > g.ny) return;
  const int r = J - 1;
  if (I >= 1) ux1[ix(g, r, I - 1)] += ux[ix(g, r, I - 1)];
  uy1[ix(g, r, I)] += uy[ix(g, r, I)];
  vof1[ix(g, r, I)] += vof[ix(g, r, I)];
}

// ---- boundary kernels of the fine-grained entry points (one thread per row)
__global__ void k_bc_ux(Grid g, double *ux) {
  pdl_entry();
  const int J = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (J > g.ny) return;
  ux[ix(g, J - 1, 0)] = 0.;
  ux[ix(g, J - 1, g.nx)] = 0.;
}
__global__ void k_bc_uy(Grid g, double *uy) {
  pdl_entry();
  const int J = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (J > g.ny) return;
  uy[ix(g, J - 1, 0)] = 0.;
  uy[ix(g, J - 1, g.nx + 1)] = 0.;
}
__global__ void k_bc_neumann(Grid g, double *f) {
  pdl_entry();
  const int J = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (J > g.ny) return;
  f[ix(g, J - 1, 0)] = f[ix(g, J - 1, 1)];
  f[ix(g, J - 1, g.nx + 1)] = f[ix(g, J - 1, g.nx)];
}
__global__ void k_bc_vof(Grid g, double *vof) {
  pdl_entry();
  const int J = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (J > g.ny) return;
  vof[ix(g, J - 1, 0)] = 0.;
  vof[ix(g, J - 1, g.nx + 1)] = 0.;
}

// test hook: the Newton-Raphson reciprocal and inverse square root on n inputs
__global__ void k_nr_check(const double *__restrict__ x, double *__restrict__ rcp, double *__restrict__ rsq, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  rcp[i] = rcp_nr(x[i]);
  rsq[i] = rsqrt_nr(x[i]);
}

// columns per transform block before tuning: with 2, 256 threads and 32 KB
// at ny = 1024, five blocks share an SM (40 warps); with 4, three (24 warps).
// The 2048 x 1024 swarm stepped 3% faster and 1024 x 512 11% faster.
constexpr int kFftCols = 2;
// dynamic shared memory of k_poisson_tdm<false> (its static xch lies beside)
constexpr size_t kTdmSmemMax = 227 * 1024 - 4096;

// FP64 fused multiply-add throughput: 8 independent chains per thread, every
// thread writes only its own output element
__global__ void k_fp64_peak(double *out, int iters, double seed) {
  const double m = 0.999999, c = 1e-7;
  double a[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) a[j] = seed + 1e-3 * j + 1e-9 * threadIdx.x;
  for (int it = 0; it < iters; ++it) {
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = fma(a[j], m, c);
  }
  double s = 0.;
#pragma unroll
  for (int j = 0; j < 8; ++j) s += a[j];
  out[(size_t)blockIdx.x * blockDim.x + threadIdx.x] = s;
}

}  // namespace

cudaError_t measure_fp64_peak(double *gflops) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int blocks = sms * 8, threads = 256, iters = 8192;
  double *out = nullptr;
  cudaError_t e = cudaMalloc(&out, sizeof(double) * blocks * threads);
  if (e != cudaSuccess) return e;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  for (int w = 0; w < 3; ++w) k_fp64_peak<<<blocks, threads>>>(out, iters, 0.1);
  float best = 1e30f;
  for (int r = 0; r < 5; ++r) {
    cudaEventRecord(e0);
    k_fp64_peak<<<blocks, threads>>>(out, iters, 0.1);
    cudaEventRecord(e1);
    cudaEventSynchronize(e1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    best = ms < best ? ms : best;
  }
  e = cudaGetLastError();
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(out);
  *gflops = 2.0 * 8.0 * blocks * threads * (double)iters / (best * 1e-3) / 1e9;
  return e;
}

cudaError_t nr_check(const double *x, double *rcp, double *rsq, int n) {
  k_nr_check<<<(n + 255) / 256, 256>>>(x, rcp, rsq, n);
  return cudaDeviceSynchronize();
}

// ===========================================================================
// launch helpers
// ===========================================================================

// columns per block of the transforms: kFftCols, halved while a block's two
// ny/2 complex rows per column exceed shared memory (ny = 8192 takes 1)
int poisson_fft_cols(int ny) {
  int w = kFftCols;
  while (w > 1 && !fft_w_fits(ny, w)) w >>= 1;
  return w;
}
size_t poisson_fft_smem(int ny, int w) { return sizeof(double2) * 2 * w * (size_t)(ny / 2); }
bool fft_w_fits(int ny, int w) { return poisson_fft_smem(ny, w) <= 227 * 1024; }

int compaction(const Tiles &t) { return g_compact >= 0 ? g_compact : t.compact; }

Tiles default_tiles(int ny) {
  Tiles t{};
  for (int k = 0; k < TK_COUNT; ++k) {
    t.bx[k] = BX;
    t.by[k] = BY;
  }
  t.fft_w = poisson_fft_cols(ny);
  t.tdm_mb = 0;
  t.tdm_g = 1;
  t.compact = 1;
  t.tdm_cl = 1;
  return t;
}
int tdm_chunk(int nx, int G) { return (nx + 32 * G - 1) / (32 * G); }
int tdm_stride(int nx, int G) { return tdm_chunk(nx, G) | 1; }
int poisson_tdm_modes(int nx) {
  const size_t per_mode = 4 * 32 * (size_t)tdm_stride(nx, 1) * sizeof(double);
  return per_mode * 4 <= 200 * 1024 ? 4 : (per_mode * 2 <= 200 * 1024 ? 2 : 1);
}
// mb: wavenumber pairs (p, M - p) per block, four systems each
size_t poisson_tdm_smem(int nx, int mb, int G) {
  return 4 * 32 * (size_t)G * tdm_stride(nx, G) * sizeof(double) * mb;
}
size_t poisson_tdm_smem(int nx) { return poisson_tdm_smem(nx, poisson_tdm_modes(nx), 1); }
bool tdm_global_stage(int nx, int G) { return poisson_tdm_smem(nx, 1, G) > kTdmSmemMax; }
size_t tdm_stage_doubles(int nx, int ny, int nc, int G) {
  return tdm_global_stage(nx, G) ? (size_t)(ny / 4 + 1) * nc * 4 * 32 * G * tdm_stride(nx, G) : 0;
}
int tdm_group_index(int G) { return G == 4 ? 2 : (G == 2 ? 1 : 0); }
// warps per tridiagonal system for a grid of nc cases: the fewest (1, 2, 4)
// that put about 2048 warps in flight (13 per SM), as long as every lane
// keeps at least 4 rows (with 2, the cross-warp combine costs more than the
// shorter recurrences save; 4 rows a lane beat 8 and 16 on every grid from
// 256 x 128 to 1024 x 512; on the 2048 x 1024 swarm 4 warps a system in
// clusters balance the SMs better but add 6% to the solve's FP64 work, and
// the step gains nothing: the side stream fills the SMs a block-per-pair
// launch leaves idle).  At 4 warps a system, and at 2 while the pairs leave
// SMs idle, the solves of a pair run as a cluster of as many CTAs
// (k_poisson_tdm_cl).  A rule of the grid, not a tuned choice: it sets how
// the chunk maps are combined, and so the rounding of the solve.
int tdm_modes_per_block(const Tiles &t, int nx) {
  const int G = t.tdm_g > 0 ? t.tdm_g : 1;
  const int mb = t.tdm_mb > 0 ? t.tdm_mb : poisson_tdm_modes(nx);
  return mb * G > 4 ? 4 / G : mb;  // at most 512 threads a block
}
// Whether the stencils of a launch over these cells share their arithmetic
// with the integer pipes: only where enough warps are in
// flight to keep the FP64 unit busy; below that an integer form's longer
// chain of instructions sets a warp's time.  Measured, us a launch, one part
// a thread on the FP64 unit, shared, and both parts shared: k_momflux 256 x
// 128 5.0, 4.5, 6.5; 500 x 128 6.7, 6.0, 7.1; 509 x 256 9.3, 8.0, 8.8; 512 x
// 512 16.2, 12.8, 13.4; k_predict_mf 6.7, 6.1, 8.4; 9.0, 8.5, 9.6; 12.8, 13.0,
// 13.3; 20.6, 21.0, 19.2.  The lines follow the whole step, whose side stream
// runs beside the predictor: us with one part on the FP64 unit and shared, 256
// x 128 113.7, 115.9; 500 x 128 160.0, 153.6; 509 x 256 244.6, 237.3, and
// 220.3 with both shared.
long cells(const Grid &g) { return (long)g.nx * g.ny * g.nc; }
bool integer_stencils(const Grid &g) { return cells(g) >= 3L << 15; }
MomHow stencil_how(const Grid &g) {
  return integer_stencils(g) ? kMomWhole : (cells(g) >= 3L << 14 ? kMomSplitInt : kMomSplit);
}
// the transforms and tridiagonal solves of smaller launches stay on the FP64 unit
bool integer_launch(const Grid &g) { return cells(g) >= 1L << 18; }
// of a transform launch with w columns a block: blocks, and complex rows, on the SM with most
long blocks_per_sm(const Grid &g, int w) { return ((long)((g.nx + w - 1) / w) * g.nc + 151) / 152; }
long rows_per_sm(const Grid &g, int w) { return w * (g.ny / 2) * blocks_per_sm(g, w); }
// The FP64 form's registers (60 to 64) leave four blocks an SM; at 48 five are resident, and up to 24 bytes spilled
// make a block itself slower: forward, 250 cases of 64 x 64 (53 blocks an SM) 59 us and with four resident 67, but
// 210 x 1024 (a block an SM or none) 20.8 us and at 60 registers 19.8
bool five_blocks(const Grid &g, int w) { return blocks_per_sm(g, w) > 4; }
// A block of w columns has w M / 4 butterflies a stage (M = ny / 2): short
// blocks have one to two warps of them, whose chain of instructions the
// integer forms lengthen, and keep the FP64 unit busy from more blocks an SM
// instead (five; the forms' registers leave four).  k_poisson_fwd and _inv,
// us, shared and alone: 250 cases of 64 x 64 73.6, 65.6 and 59.2, 51.8; 32 of
// 256 x 128 42.0, 34.8 and 35.4, 31.5; 8 of 512 x 256 38.7, 32.7 and 33.7,
// 28.7; 20 of 100 x 512 32.9, 26.2 and 34.7, 28.7; 4 of 300 x 1024 37.9, 30.5
// and 44.4, 35.3.  With few blocks an SM both wait for loads and barriers, and
// what counts is the FP64 unit's time left to the side stream: the step of 512
// x 512 (two blocks an SM) 287 and 272 us, of 800 x 512 (three) 362 and 372.
bool integer_transforms(const Grid &g, int w) {
  return integer_launch(g) && w * (g.ny / 2) >= 512 && rows_per_sm(g, w) >= 1536;
}
// Chunks of L rows: the integer forms' registers (94, plainly 60) and groups of
// kAhead rows pay for long ones.  k_poisson_tdm, us, shared and plainly: 1000
// cases of 32 x 32 (1 row) 203 and 88, 250 of 64 x 64 (2) 102 and 56, 128 of
// 128 x 64 (4) 63 and 47, 64 of 224 x 128 (7) 64 and 60; the step of 32 cases
// of 256 x 128 (8) 846 and 861 us.  Where few pairs are spread over warps (G >
// 1) the loads ahead count from 5 rows on: 600 x 512 21.6 and 22.4 us, 600 x
// 1024 (10) 26.3 and 27.6, its step 487 and 524.  Registers pay for a launch
// of less than two blocks an SM: 256 x 128 (33 pairs, 4 rows) 12.3 us and
// plainly 14.3, 13 cases of 128 x 64 (221) 12.1 and 12.5; 30 of 64 x 64 (510, 2
// rows) 14.2 and 13.0; the step of 100 cases of 16 x 8 (300, 1 row) 122 and 112.
TdmHow tdm_how(const Grid &g, int G) {
  const int L = tdm_chunk(g.nx, G);
  if (integer_launch(g) && L >= (G > 1 ? 5 : 8)) return kTdmInt;
  const long pairs = (g.ny / 4 + 1L) * g.nc;
  return L <= kTdmRegRows && pairs < (L >= 3 ? 304 : 152) ? kTdmReg : kTdmPlain;
}
// Whether a launch spreads its butterflies over lanes: its warps issue twice
// the FP64 instructions, in a quarter of the turns, so it pays while they are
// few enough a scheduler, W M complex rows a block and that many blocks an SM
// making at most 256.  Measured, us a launch of k_poisson_fwd: 64 x 64 (64)
// 6.7 -> 4.8, 256 x 128 (128) 7.2 -> 5.8, 256 x 256 (256) 8.9 -> 8.7, 509 x
// 256 (512) 9.3 -> 10.4, 128 x 1024 (1024) 17.1 -> 27.6.
bool lane_transforms(const Grid &g, int w) { return rows_per_sm(g, w) <= 256; }
// default pairs per block: as many as shared memory and 512 threads take, but
// one block a pair while the pairs are too few to give every SM that many
// (its warps share one FP64 unit a scheduler: 64 x 64 k_poisson_tdm 10.8 ->
// 7.8 us, 256 x 128 15.7 -> 11.9 us)
int tdm_modes_for(int nx, int ny, int nc, int G) {
  const long pairs = (long)(ny / 4 + 1) * nc;
  int mb = std::min(poisson_tdm_modes(nx), 4 / G);
  while (mb > 1 && pairs < 152L * mb) mb >>= 1;
  return mb;
}
int tdm_warps_for(int nx, int ny, int nc) {
  const long systems = 4L * (ny / 4 + 1) * nc;
  int G = 1;
  while (G < 4 && systems * G < 2048 && tdm_chunk(nx, 2 * G) >= 4) G *= 2;
  return G;
}

template <class... K>
cudaError_t allow_smem(int bytes, K... kernels) {
  cudaError_t e = cudaSuccess;
  ((e = e == cudaSuccess ? cudaFuncSetAttribute(kernels, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) : e), ...);
  return e;
}
template <int... W>
cudaError_t configure_fft(int bytes) {
  const cudaError_t e =
      allow_smem(bytes, k_poisson_fwd<1, false, kFftLanes>, k_poisson_fwd<2, false, kFftLanes>,
                 k_poisson_fwd<1, true, kFftLanes>, k_poisson_fwd<2, true, kFftLanes>, k_poisson_inv<1, kFftLanes>,
                 k_poisson_inv<2, kFftLanes>);
  if (e != cudaSuccess) return e;
  return allow_smem(bytes, k_poisson_fwd<W, false, kFftPlain>..., k_poisson_fwd<W, true, kFftPlain>...,
                    k_poisson_fwd<W, false, kFftInt>..., k_poisson_fwd<W, true, kFftInt>...,
                    k_poisson_fwd<W, false, kFftShort>..., k_poisson_fwd<W, true, kFftShort>...,
                    k_poisson_inv<W, kFftPlain>..., k_poisson_inv<W, kFftInt>..., k_poisson_inv<W, kFftShort>...);
}

cudaError_t configure_kernels() {
  cudaError_t e;
  const int big = 227 * 1024;
  e = configure_fft<1, 2, 4, 8>(big);
  if (e != cudaSuccess) return e;
  return allow_smem((int)kTdmSmemMax, k_poisson_tdm<false, kTdmPlain>, k_poisson_tdm<false, kTdmReg>,
                    k_poisson_tdm<false, kTdmInt>, k_poisson_tdm_cl<kTdmPlain, 2>, k_poisson_tdm_cl<kTdmReg, 2>,
                    k_poisson_tdm_cl<kTdmInt, 2>, k_poisson_tdm_cl<kTdmPlain, 4>, k_poisson_tdm_cl<kTdmReg, 4>,
                    k_poisson_tdm_cl<kTdmInt, 4>);
}

void launch_props(cudaStream_t s, const Grid &g, const Metrics &m, const Phys &ph, const Bufs &b, bool den, bool vis,
                  bool grad, double *den_out, bool scaled) {
  const dim3 gr = tile_grid(b.tiles, TK_PROPS, g.nx + 2, g.ny, g.nc), bl = tile_block(b.tiles, TK_PROPS);
  int *counts = vis && grad ? b.icount : nullptr;  // a step's: the geometry follows
  if (scaled && vis && grad && !den)
    launch_pdl(k_props<false, true, true, true>, gr, bl, 0, s, g, m, ph, b.vof, den_out, b.visux, b.visuy, b.dvof,
               compaction(b.tiles), counts);
  else if (den && vis && grad)
    launch_pdl(k_props<true, true, true>, gr, bl, 0, s, g, m, ph, b.vof, den_out, b.visux, b.visuy, b.dvof,
               compaction(b.tiles), counts);
  else if (vis && grad)
    launch_pdl(k_props<false, true, true>, gr, bl, 0, s, g, m, ph, b.vof, den_out, b.visux, b.visuy, b.dvof,
               compaction(b.tiles), counts);
  else if (den)
    launch_pdl(k_props<true, false, false>, gr, bl, 0, s, g, m, ph, b.vof, den_out, b.visux, b.visuy, b.dvof,
               compaction(b.tiles), counts);
  else if (vis)
    launch_pdl(k_props<false, true, false>, gr, bl, 0, s, g, m, ph, b.vof, den_out, b.visux, b.visuy, b.dvof,
               compaction(b.tiles), counts);
  else if (grad)
    launch_pdl(k_props<false, false, true>, gr, bl, 0, s, g, m, ph, b.vof, den_out, b.visux, b.visuy, b.dvof,
               compaction(b.tiles), counts);
}

void launch_normal_curv(cudaStream_t s, const Grid &g, const Metrics &m, const Bufs &b, bool normal, bool curv,
                        bool store_k) {
  const dim3 gr = grid2d(g.nx, g.ny), bl(BX, BY);
  if (normal && curv && store_k)
    launch_pdl(k_normal_curv<true, true, true>, gr, bl, 0, s, g, m, b.vof, b.dvof, b.normal, b.curv);
  else if (normal && curv)
    launch_pdl(k_normal_curv<true, true, false>, gr, bl, 0, s, g, m, b.vof, b.dvof, b.normal, b.curv);
  else if (normal)
    launch_pdl(k_normal_curv<true, false, false>, gr, bl, 0, s, g, m, b.vof, b.dvof, b.normal, b.curv);
  else if (curv)
    launch_pdl(k_normal_curv<false, true, false>, gr, bl, 0, s, g, m, b.vof, b.dvof, b.normal, b.curv);
}

void launch_flux_force(cudaStream_t s, const Grid &g, const Metrics &m, const Phys &ph, const Bufs &b,
                       const double *ux, const double *uy, const double *den0, bool flux, bool force, bool have_k) {
  const dim3 gr = grid2d(g.nx, g.ny), bl(BX, BY);
  if (flux && force && have_k)
    launch_pdl(k_flux_force<true, true, true>, gr, bl, 0, s, g, m, ph, ux, uy, b.vof, b.normal, den0, b.curv, b.fluxx,
                                                     b.fluxy, b.ifrcx, b.ifrcy);
  else if (flux && force)
    launch_pdl(k_flux_force<true, true, false>, gr, bl, 0, s, g, m, ph, ux, uy, b.vof, b.normal, den0, b.curv, b.fluxx,
                                                      b.fluxy, b.ifrcx, b.ifrcy);
  else if (flux)
    launch_pdl(k_flux_force<true, false, false>, gr, bl, 0, s, g, m, ph, ux, uy, b.vof, b.normal, den0, b.curv, b.fluxx,
                                                       b.fluxy, b.ifrcx, b.ifrcy);
  else if (force)
    launch_pdl(k_flux_force<false, true, false>, gr, bl, 0, s, g, m, ph, ux, uy, b.vof, b.normal, den0, b.curv, b.fluxx,
                                                       b.fluxy, b.ifrcx, b.ifrcy);
}

void launch_interface_stage(cudaStream_t s, const Grid &g, const Metrics &m, const Phys &ph, const Bufs &b,
                            const double *ux, const double *uy, const double *den0, int stage) {
  const dim3 gr = tile_grid(b.tiles, TK_FLUX_FORCE, g.nx, g.ny, g.nc), bl = tile_block(b.tiles, TK_FLUX_FORCE);
  if (stage == 0) {
    launch_pdl(k_curv_list<true>, tile_grid(b.tiles, TK_CURV_LIST, g.nx, g.ny, g.nc), tile_block(b.tiles, TK_CURV_LIST),
               0, s, g, m, b.vof, b.dvof, ux, uy, b.curv, b.ilist, b.icount, b.flist, b.fcount, (double *)nullptr,
               compaction(b.tiles));
  } else if (stage == 1) {
    launch_pdl(k_interface_cells, dim3(max(2, (4 * 152 + g.nc - 1) / g.nc), 1, g.nc), 256, 0, s,
        g, m, ux, uy, b.vof, b.dvof, b.flist, b.fcount, b.fluxx, b.fluxy);
  } else if (stage == 2) {
    launch_pdl(k_flux_force<true, true, true, true>, gr, bl, 0, s, g, m, ph, ux, uy, b.vof, b.normal, den0, b.curv, b.fluxx,
                                                           b.fluxy, b.ifrcx, b.ifrcy);
  } else {
    launch_pdl(k_flux_force<true, true, true, true, true>, gr, bl, 0, s, g, m, ph, ux, uy, b.vof, b.normal, den0, b.curv,
                                                                 b.fluxx, b.fluxy, b.ifrcx, b.ifrcy);
  }
}

// An SM takes blocks of another kernel only under the split of its memory that
// it has: the geometry's blocks beside a short transform's, whose split is
// smaller, all went to the few SMs without one of those (40 blocks to five
// SMs, eight on each: 30 us instead of 6).
// On grids that short, while there is an SM for every block, they ask for the
// smallest split that holds one (in percent): ten cases of 32 x 32, a step 161
// -> 92 us, of 64 x 32 147 -> 99 us, of 48 x 32 137 -> 96 us.  Elsewhere the
// smaller split costs more than the crowding (24 cases of 64 x 32 145 and 160
// us, 4 of 128 x 64 108 and 115, 509 x 256 183 and 201).
constexpr int kFewBlocksSmem = 3;
void launch_geometry(cudaStream_t s, const Grid &g, const Metrics &m, const Bufs &b) {
  const dim3 gr = tile_grid(b.tiles, TK_CURV_LIST, g.nx, g.ny, g.nc);
  const bool few = g.ny <= 32 && (long)gr.x * gr.y * gr.z <= 152;
  launch_pdl_smem(few ? kFewBlocksSmem : -1, k_curv_list<false>, gr, tile_block(b.tiles, TK_CURV_LIST), 0, s, g, m, b.vof,
                  b.dvof, (const double *)nullptr, (const double *)nullptr, b.curv, b.ilist, b.icount, b.flist, b.fcount,
                  b.tf, compaction(b.tiles));
}

void launch_bulk_flux(cudaStream_t s, const Grid &g, const Metrics &m, const Phys &ph, const Bufs &b,
                      const double *ux, const double *uy) {
  launch_pdl(k_bulk_flux, tile_grid(b.tiles, TK_FLUX_FORCE, g.nx, g.ny, g.nc), tile_block(b.tiles, TK_FLUX_FORCE), 0, s,
             g, m, ph, ux, uy, b.vof, b.fluxx, b.fluxy);
}

void launch_csf_force(cudaStream_t s, const Grid &g, const Metrics &m, const Phys &ph, const Bufs &b,
                      const double *den0, double *ifx, double *ify, bool itf_kappa) {
  const dim3 gr = tile_grid(b.tiles, TK_FORCE, g.nx, g.ny, g.nc), bl = tile_block(b.tiles, TK_FORCE);
  if (itf_kappa)
    launch_pdl(k_csf_force<true>, gr, bl, 0, s, g, m, ph, b.vof, den0, b.curv, ifx, ify);
  else
    launch_pdl(k_csf_force<false>, gr, bl, 0, s, g, m, ph, b.vof, den0, b.curv, ifx, ify);
}

void launch_vof_advance(cudaStream_t s, const Grid &g, const Metrics &m, const Phys &ph, const Bufs &b,
                        const double *sc, int k, double *src_a, const double *src_b, bool fused, const double *ux,
                        const double *uy, double *den1, double *vof_out) {
  const dim3 gr = tile_grid(b.tiles, TK_VOF_ADVANCE, g.nx, g.ny, g.nc), bl = tile_block(b.tiles, TK_VOF_ADVANCE);
  if (fused && vof_out)
    launch_pdl(integer_stencils(g) ? k_vof_advance<true, true, true> : k_vof_advance<true, true, false>, gr, bl, 0, s, g, m,
               ph, sc, k, b.vof, vof_out, b.fluxx, b.fluxy, src_a, src_b,
               ux, uy, b.mfluxx, b.mfluxy, den1);
  else if (fused)
    launch_pdl(k_vof_advance<true, false, false>, gr, bl, 0, s, g, m, ph, sc, k, b.vof, (double *)nullptr, b.fluxx, b.fluxy,
               src_a, src_b, ux, uy, b.mfluxx, b.mfluxy, den1);
  else
    launch_pdl(k_vof_advance<false, false, false>, gr, bl, 0, s, g, m, ph, sc, k, b.vof, (double *)nullptr, b.fluxx, b.fluxy,
               src_a, src_b, ux, uy, (double *)nullptr, (double *)nullptr, (double *)nullptr);
}

void launch_face_flux(cudaStream_t s, const Grid &g, const Bufs &b, const double *ux, const double *uy) {
  launch_pdl(k_face_flux, dim3(max(2, (4 * 152 + g.nc - 1) / g.nc), 1, g.nc), 256, 0, s, g, ux, uy, b.ilist, b.icount,
             b.tf, b.fluxx, b.fluxy);
}

void launch_mass_flux_inplace(cudaStream_t s, const Grid &g, const Phys &ph, const Bufs &b, const double *ux,
                              const double *uy) {
  launch_pdl(k_mass_flux, grid2d(g.nx + 2, g.ny), dim3(BX, BY), 0, s, g, ph, ux, uy, b.fluxx, b.fluxy);
}

void launch_stress(cudaStream_t s, const Grid &g, const Metrics &m, const Bufs &b, const double *ux,
                   const double *uy) {
  launch_pdl(k_stress, tile_grid(b.tiles, TK_MOMFLUX, g.nx + 1, g.ny, g.nc), tile_block(b.tiles, TK_MOMFLUX), 0, s, g,
             m, ux, uy, b.visux, b.visuy, b.txx, b.txy, b.tyy);
}

void launch_momflux(cudaStream_t s, const Grid &g, const Metrics &m, const Phys &ph, const Bufs &b,
                    const double *ux, const double *uy, int stress, bool scaled) {
  dim3 gr = tile_grid(b.tiles, TK_MOMFLUX, g.nx + 1, g.ny, g.nc), bl = tile_block(b.tiles, TK_MOMFLUX);
  auto k = k_momflux<2, false, kMomWhole>;
  if (stress != 2 && !scaled) k = stress == 1 ? k_momflux<1, false, kMomWhole> : k_momflux<0, false, kMomWhole>;
  if (stress != 2 && scaled) {
    const MomHow how = stencil_how(g);
    if (how == kMomWhole)
      k = stress == 1 ? k_momflux<1, true, kMomWhole> : k_momflux<0, true, kMomWhole>;
    else if (how == kMomSplitInt)
      k = stress == 1 ? k_momflux<1, true, kMomSplitInt> : k_momflux<0, true, kMomSplitInt>;
    else
      k = stress == 1 ? k_momflux<1, true, kMomSplit> : k_momflux<0, true, kMomSplit>;
    if (how != kMomWhole) gr.y *= 2;
  }
  launch_pdl(k, gr, bl, 0, s, g, m, ph, (const double *)b.scalars, ux, uy, b.visux, b.visuy, b.mfluxx, b.mfluxy, b.pxx, b.pyy, b.pxy, b.pyx,
             b.txx, b.txy, b.tyy);
}

void launch_predict_mf(cudaStream_t s, const Grid &g, const Metrics &m, const Phys &ph, const Bufs &b,
                       const double *sc, int k, const double *ux, const double *uy, double *ux_out, double *uy_out,
                       const double *den0, const double *den1, const double *psi_old, double *srcux_a,
                       const double *srcux_b, double *srcuy_a, const double *srcuy_b, const double *ifx,
                       const double *ify, bool cached) {
  const MomHow how = stencil_how(g);
  auto kern = cached ? k_predict_mf<true, kMomSplit> : k_predict_mf<false, kMomSplit>;
  if (how == kMomSplitInt) kern = cached ? k_predict_mf<true, kMomSplitInt> : k_predict_mf<false, kMomSplitInt>;
  if (how == kMomWhole) kern = cached ? k_predict_mf<true, kMomWhole> : k_predict_mf<false, kMomWhole>;
  dim3 gr = tile_grid(b.tiles, TK_PREDICT, g.nx, g.ny, g.nc);
  if (how != kMomWhole) gr.y *= 2;
  launch_pdl(kern, gr, tile_block(b.tiles, TK_PREDICT), 0, s, g, m, ph,
             sc, k, ux, uy, ux_out, uy_out, b.pxx, b.pyy, b.pxy, b.pyx, b.p, ifx, ify, den0, den1, psi_old, srcux_a,
             srcux_b, srcuy_a, srcuy_b, b.egx, b.egy, b.coltab, b.qx, b.qy, b.rhofx, b.rhofy, b.dpsix, b.dpsiy);
}

void launch_predict(cudaStream_t s, const Grid &g, const Metrics &m, const Phys &ph, const Bufs &b, const double *sc,
                    int k, const double *ux, const double *uy, double *ux_out, double *uy_out, const double *mfx,
                    const double *mfy, const double *den0, const double *den1, double *srcux_a,
                    const double *srcux_b, double *srcux_g, double *srcuy_a, const double *srcuy_b,
                    double *srcuy_g) {
  launch_pdl(k_predict, tile_grid(b.tiles, TK_PREDICT, g.nx, g.ny, g.nc), tile_block(b.tiles, TK_PREDICT), 0, s, g, m, ph, sc, k, ux, uy, ux_out, uy_out, mfx, mfy, b.txx,
                                                        b.txy, b.tyy, b.p, b.ifrcx, b.ifrcy, den0, den1, srcux_a,
                                                        srcux_b, srcux_g, srcuy_a, srcuy_b, srcuy_g);
}

template <int W, bool Q>
void poisson_fwd_w(cudaStream_t s, const Grid &g, const Bufs &b, const double *sc, int k, const double *ux,
                   const double *uy) {
  const int nb = (g.nx + W - 1) / W;
  auto kern = five_blocks(g, W) ? k_poisson_fwd<W, Q, kFftShort> : k_poisson_fwd<W, Q, kFftPlain>;
  if (integer_transforms(g, W)) kern = k_poisson_fwd<W, Q, kFftInt>;
  if (W <= 2 && lane_transforms(g, W)) kern = k_poisson_fwd<(W <= 2 ? W : 2), Q, kFftLanes>;
  launch_pdl(kern, dim3(nb, 1, g.nc), 256, poisson_fft_smem(g.ny, W), s, g, sc, k, ux, uy, b.egx, b.egy, b.twiddle, b.spec);
}

template <bool Q>
void poisson_fwd_any(cudaStream_t s, const Grid &g, const Bufs &b, const double *sc, int k, const double *ux,
                     const double *uy) {
  if (b.tiles.fft_w == 1)
    poisson_fwd_w<1, Q>(s, g, b, sc, k, ux, uy);
  else if (b.tiles.fft_w == 2)
    poisson_fwd_w<2, Q>(s, g, b, sc, k, ux, uy);
  else if (b.tiles.fft_w == 8)
    poisson_fwd_w<8, Q>(s, g, b, sc, k, ux, uy);
  else
    poisson_fwd_w<4, Q>(s, g, b, sc, k, ux, uy);
}

void launch_poisson_fwd(cudaStream_t s, const Grid &g, const Bufs &b, const double *sc, int k, const double *ux,
                        const double *uy) {
  poisson_fwd_any<false>(s, g, b, sc, k, ux, uy);
}

void launch_poisson_fwd_q(cudaStream_t s, const Grid &g, const Bufs &b, const double *sc, int k) {
  poisson_fwd_any<true>(s, g, b, sc, k, b.qx, b.qy);
}

int g_tdm_cluster = 1;

bool tdm_uses_cluster(const Tiles &t, int nx) {
  return g_tdm_cluster && t.tdm_cl && t.tdm_g >= 2 &&
         4 * 32 * (size_t)tdm_stride(nx, t.tdm_g) * sizeof(double) <= kTdmSmemMax;
}

template <int CL>
auto tdm_cluster_kernel(TdmHow how) {
  return how == kTdmInt ? k_poisson_tdm_cl<kTdmInt, CL>
                        : (how == kTdmReg ? k_poisson_tdm_cl<kTdmReg, CL> : k_poisson_tdm_cl<kTdmPlain, CL>);
}

void launch_poisson_tdm(cudaStream_t s, const Grid &g, const Bufs &b) {
  const int G = b.tiles.tdm_g > 0 ? b.tiles.tdm_g : 1;
  const int pairs = g.ny / 4 + 1, L = tdm_chunk(g.nx, G), S = tdm_stride(g.nx, G);
  const double4_32a *fac = reinterpret_cast<const double4_32a *>(b.tdm_fac[tdm_group_index(G)]);
  const TdmHow how = tdm_how(g, G);
  if (tdm_uses_cluster(b.tiles, g.nx)) {  // G CTAs per pair, four warps each
    launch_pdl(G == 4 ? tdm_cluster_kernel<4>(how) : tdm_cluster_kernel<2>(how), dim3(G * pairs, 1, g.nc), 128,
               4 * 32 * (size_t)S * sizeof(double), s, g, L, S, fac, b.twiddle, b.spec);
    return;
  }
  if (tdm_global_stage(g.nx, G)) {  // one pair per block, staged in b.tdm_stage
    launch_pdl(how == kTdmInt ? k_poisson_tdm<true, kTdmInt> : k_poisson_tdm<true, kTdmPlain>, dim3(pairs, 1, g.nc),
               128 * G, 0, s, g, 1, G, L, S, fac, b.twiddle, b.spec, b.tdm_stage);
    return;
  }
  const int mb = tdm_modes_per_block(b.tiles, g.nx);  // wavenumber pairs per block
  auto kern = how == kTdmInt ? k_poisson_tdm<false, kTdmInt>
                             : (how == kTdmReg ? k_poisson_tdm<false, kTdmReg> : k_poisson_tdm<false, kTdmPlain>);
  launch_pdl(kern, dim3((pairs + mb - 1) / mb, 1, g.nc), 128 * mb * G, poisson_tdm_smem(g.nx, mb, G), s, g, mb, G, L, S, fac,
             b.twiddle, b.spec, (double *)nullptr);
}

template <int W>
void poisson_inv_w(cudaStream_t s, const Grid &g, const Bufs &b, double *psi_new) {
  const int nb = (g.nx + W - 1) / W;
  auto kern = five_blocks(g, W) ? k_poisson_inv<W, kFftShort> : k_poisson_inv<W, kFftPlain>;
  if (integer_transforms(g, W)) kern = k_poisson_inv<W, kFftInt>;
  if (W <= 2 && lane_transforms(g, W)) kern = k_poisson_inv<(W <= 2 ? W : 2), kFftLanes>;
  launch_pdl(kern, dim3(nb, 1, g.nc), 256, poisson_fft_smem(g.ny, W), s, g, b.twiddle, b.spec, psi_new);
}

void launch_poisson_inv(cudaStream_t s, const Grid &g, const Bufs &b, double *psi_new) {
  if (b.tiles.fft_w == 1)
    poisson_inv_w<1>(s, g, b, psi_new);
  else if (b.tiles.fft_w == 2)
    poisson_inv_w<2>(s, g, b, psi_new);
  else if (b.tiles.fft_w == 8)
    poisson_inv_w<8>(s, g, b, psi_new);
  else
    poisson_inv_w<4>(s, g, b, psi_new);
}

void launch_poisson(cudaStream_t s, const Grid &g, const Bufs &b, const double *sc, int k, const double *ux,
                    const double *uy, double *psi_new) {
  launch_poisson_fwd(s, g, b, sc, k, ux, uy);
  launch_poisson_tdm(s, g, b);
  launch_poisson_inv(s, g, b, psi_new);
}

void launch_correct(cudaStream_t s, const Grid &g, const Metrics &m, const Bufs &b, const double *sc, int k,
                    double *ux, double *uy, const double *psi_new, bool pressure, bool dpsi) {
  const dim3 gr = tile_grid(b.tiles, TK_CORRECT, g.nx, g.ny, g.nc), bl = tile_block(b.tiles, TK_CORRECT);
  auto kern = pressure ? (dpsi ? k_correct<true, true> : k_correct<true, false>)
                       : (dpsi ? k_correct<false, true> : k_correct<false, false>);
  launch_pdl(kern, gr, bl, 0, s, g, sc, b.coltab, k, ux, uy, psi_new, b.egx, b.egy, b.p, b.dpsix, b.dpsiy);
}

void launch_pressure(cudaStream_t s, const Grid &g, const Bufs &b, const double *psi_new) {
  launch_pdl(k_pressure, grid2d(g.nx, g.ny), dim3(BX, BY), 0, s, g, psi_new, b.p);
}

void launch_decide_dt(cudaStream_t s, const Grid &g, const Metrics &m, const Phys &ph, const Bufs &b,
                      const double *ux, const double *uy, double dt_fixed, double coef_adv) {
  launch_decide_dt_raw(s, g, m, ph, ux, uy, b.dt_acc, b.scalars, b.status, dt_fixed, coef_adv, b.coltab);
}

void launch_decide_dt_raw(cudaStream_t s, const Grid &g, const Metrics &m, const Phys &ph, const double *ux,
                          const double *uy, unsigned long long *acc, double *sc, int *status, double dt_fixed,
                          double coef_adv, double *coltab) {
  int gy = (g.ny + BY - 1) / BY;
  const int gx = (g.nx + BX) / BX;
  while (gy > 1 && gx * gy * g.nc > 16 * 152) gy = (gy + 1) / 2;
  launch_pdl(k_decide_dt, dim3(gx, gy, g.nc), dim3(BX, BY), 0, s, g, ux, uy, acc);
  launch_pdl(k_decide_dt_fin, dim3((g.nx + kDtFinThreads - 1) / kDtFinThreads, 1, g.nc), dim3(kDtFinThreads), 0, s, g, m,
             ph, acc, sc, status, dt_fixed, coef_adv);
  if (coltab) launch_decide_dt_tab(s, g, m, sc, coltab);
}

void launch_decide_dt_tab(cudaStream_t s, const Grid &g, const Metrics &m, const double *sc, double *coltab) {
  launch_pdl(k_decide_dt_tab, dim3((g.nx + 2 + kDtFinThreads - 1) / kDtFinThreads, 1, g.nc), dim3(kDtFinThreads), 0, s, g,
             m, sc, coltab);
}

void launch_face_factor(cudaStream_t s, const Grid &g, const Phys &ph, const Bufs &b, const double *den,
                        const double *psi_old) {
  launch_pdl(k_face_factor, grid2d(g.nx + 1, g.ny), dim3(BX, BY), 0, s, g, b.scalars, den, psi_old, b.egx, b.egy);
}

int diag_partial_blocks(const Grid &g) {
  const dim3 gr = grid2d(g.nx, g.ny);
  return (int)(gr.x * gr.y);
}

void launch_diagnostics(cudaStream_t s, const Grid &g, const Metrics &m, const double *ux, const double *uy,
                        const double *vof, const double *den, const double *txy, double nu, double *part,
                        double *out) {
  const dim3 gr = grid2d(g.nx, g.ny);
  launch_pdl(k_diag_partial, gr, dim3(BX, BY), 0, s, g, m, ux, uy, vof, den, txy, nu, part);
  launch_pdl(k_diag_final, 1, BX * BY, 0, s, part, (int)(gr.x * gr.y), out);
}

void launch_stats_collect(cudaStream_t s, const Grid &g, const double *ux, const double *uy, const double *vof,
                          double *ux1, double *uy1, double *vof1) {
  launch_pdl(k_stats_collect, grid2d(g.nx + 2, g.ny), dim3(BX, BY), 0, s, g, ux, uy, vof, ux1, uy1, vof1);
}

void launch_bc_ux(cudaStream_t s, const Grid &g, double *ux) { launch_pdl(k_bc_ux, (g.ny + 127) / 128, 128, 0, s, g, ux); }
void launch_bc_uy(cudaStream_t s, const Grid &g, double *uy) { launch_pdl(k_bc_uy, (g.ny + 127) / 128, 128, 0, s, g, uy); }
void launch_bc_neumann(cudaStream_t s, const Grid &g, double *f) {
  launch_pdl(k_bc_neumann, (g.ny + 127) / 128, 128, 0, s, g, f);
}
void launch_bc_vof(cudaStream_t s, const Grid &g, double *vof) {
  launch_pdl(k_bc_vof, (g.ny + 127) / 128, 128, 0, s, g, vof);
}

// ---------------------------------------------------------------------------
// the caller's host arrays <-> device fields, copied by the GPU itself over
// the CPU-GPU link (host memory the device can address: pageable memory on a
// system with host page-table access, or registered memory).  In: host rows
// J = 1..ny (x ghosts included) into the pitched device rows.  Out: every host
// row J = 1 - ay0 .. ny + ay1, the y ghost rows from their periodic images
// (what the reference's halo exchange leaves there, src/halo.c:18-76).  Case
// z of a batch is blockIdx.y: its arrays are tab[z * kLinkSlots + slot], its
// device rows start at dev + z * cs1.  Each thread keeps four loads in flight:
// the link's latency is microseconds.  nwords doubles from words to
// words_host (page-locked) come along, over all blocks (64 a case: 8000 cases of
// 16 x 8, a host-linked step 10.3 ms with all on one block, 9.7 ms so).
template <bool kIn>
__global__ void __launch_bounds__(256) k_host_rows(Grid g, double *const *tab, HostRows a, HostRows b, HostRows c, int nf,
                                                   const double *words, double *words_host, int nwords) {
  pdl_entry();
  for (int t = (blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x; t < nwords;
       t += gridDim.x * gridDim.y * blockDim.x)
    words_host[t] = words[t];
  const int z = blockIdx.y;
  const int stride = gridDim.x * blockDim.x;
  for (int q = 0; q < nf; ++q) {
    const HostRows f = q == 0 ? a : (q == 1 ? b : c);
    double *h = tab[(size_t)z * kLinkSlots + f.slot];
    double *dev = f.dev + (size_t)z * g.cs1;
    const int n = (kIn ? g.ny : g.ny + f.ay0 + f.ay1) * f.row;
    for (int t0 = blockIdx.x * blockDim.x + threadIdx.x; t0 < n; t0 += 4 * stride) {
      double v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int t = t0 + u * stride;
        if (t >= n) break;
        const int r = t / f.row, i = t - r * f.row;
        // in: host row J = r + 1 (index r + ay0); out: host row index r holds J = r + 1 - ay0
        v[u] = kIn ? h[(size_t)(r + f.ay0) * f.row + i] : dev[(size_t)wrap(r - f.ay0 + 1, g.ny) * g.p1 + i];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int t = t0 + u * stride;
        if (t >= n) break;
        if (kIn) {
          const int r = t / f.row, i = t - r * f.row;
          dev[(size_t)r * g.p1 + i] = v[u];
        } else {
          h[t] = v[u];
        }
      }
    }
  }
}

void launch_host_rows(cudaStream_t s, const Grid &g, double *const *tab, bool in, HostRows a, HostRows b, int nf,
                      int width, HostRows c, const double *words, double *words_host, int nwords) {
  const dim3 grid(std::max(1, width / g.nc), g.nc);
  if (in)
    launch_pdl(k_host_rows<true>, grid, 256, 0, s, g, tab, a, b, c, nf, words, words_host, nwords);
  else
    launch_pdl(k_host_rows<false>, grid, 256, 0, s, g, tab, a, b, c, nf, words, words_host, nwords);
}

// the same for the fine-grained entry points: field blockIdx.y of the list, a
// launch instead of a copy-engine call per field and ghost row (300 x 256
// curvature call, 6 MB over the link: 192 us with five copies and eight ghost
// rows, 72 us)
template <bool kIn>
__global__ void __launch_bounds__(256) k_host_fields(const __grid_constant__ HostFields fs) {
  pdl_entry();
  const HostField &f = fs.f[blockIdx.y];
  const int stride = gridDim.x * blockDim.x;
  const int n = (kIn ? f.rows : f.rows + f.ay0 + f.ay1) * f.row;
  for (int t0 = blockIdx.x * blockDim.x + threadIdx.x; t0 < n; t0 += 4 * stride) {
    double v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int t = t0 + u * stride;
      if (t >= n) break;
      const int r = t / f.row, i = t - r * f.row;
      v[u] = kIn ? f.h[(size_t)(r + f.ay0) * f.row + i] : f.dev[wrap(r - f.ay0 + 1, f.rows) * f.pitch + i];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int t = t0 + u * stride;
      if (t >= n) break;
      const int r = t / f.row, i = t - r * f.row;
      if (kIn)
        f.dev[r * f.pitch + i] = v[u];
      else
        f.h[t] = v[u];
    }
  }
}

void launch_host_fields(cudaStream_t s, const HostFields &fs, int n, bool in) {
  const dim3 grid(std::max(16, 4 * 152 / n), n);
  if (in)
    launch_pdl(k_host_fields<true>, grid, 256, 0, s, fs);
  else
    launch_pdl(k_host_fields<false>, grid, 256, 0, s, fs);
}

}  // namespace sbfs
