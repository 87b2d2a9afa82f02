// sg_apply_mf.cu -- matrix-free FP32 element apply of the mixed form.
//
// With GLL quadrature at the 27 element nodes the stored element matrix is
//   K_e = sum_q w_q detJ_q B_q^T C B_q        (src/preprocess.f90:74-148),
// so K_e p can be formed without K_e: at every GLL point q take the gradient
// of p (each reference derivative is a 3-term sum along one lattice line,
// with the 1D GLL derivative matrix D), map it with J^-1, form the stress
// sigma = C eps with the engineering shears of compute_bmat
// (src/preprocess.f90:12-68) and the isotropic C of compute_cmat
// (src/elastic.f90:13-42), and return it through B_q^T (again 3-term line
// sums).  Per element this reads a 48-byte record per GLL point (J^-1 and the
// three C constants scaled by w_q detJ_q, 1.3 KB per element) instead of the
// 9.7 KB of stored FP32 entries, and costs about 3,600 FMAs per right-hand
// side against 4,617.
//
// Four trials and more: thread (element, plane of nine nodes, trial): the xi and eta terms of a plane
// stay in the thread's registers; only the zeta terms cross threads, through
// shared memory.  Three warps, one per plane, make a group that takes 32 / KR
// elements at a time.  What bounds it: instruction issue (some 1,100 warp
// instructions an element at 8 trials, 1,071 of each thread's 1,500 being the
// arithmetic) and behind it HBM.  Against one thread per lattice line this
// halves the shared traffic (142 wavefronts an element instead of 304) and the
// barriers cover three warps instead of the block (us per apply, line form
// before, this now: 62k elements and 8 trials 220, 134; 16k and 16 trials 128,
// 78; 36k and 4 trials 78, 52).  A group's maps and point
// records arrive by cp.async while the group before is computed, and the next
// p and z rows are on their way during the zeta pass.
//
// The FP64 residual of the mixed solve keeps the stored FP64 matrices, so this
// operator only steers the FP32 inner iterations.  It is nearer to them than their
// entries rounded to FP32 are, since the gradient takes the differences of p
// first: relative error of the element products on a 192,000-element slope 6e-8
// against 9e-8 for noise, 1e-7 against 6e-7 for a wave of an eighth of the slope,
// 9e-7 against 5e-6 for a settlement.
#include <cstdint>
#include <cstdlib>

#include "sg_kernels.cuh"

namespace sg {

namespace mf {


// D[i][t] = derivative of the 1D Lagrange basis t at GLL point i (nodes -1, 0, 1)
__device__ __forceinline__ constexpr float Dm(int i, int t) {
  return i == 0 ? (t == 0 ? -1.5f : t == 1 ? 2.0f : -0.5f)
                : i == 1 ? (t == 0 ? -0.5f : t == 1 ? 0.0f : 0.5f) : (t == 0 ? 0.5f : t == 1 ? -2.0f : 1.5f);
}

// Stress fluxes at one GLL point from the reference gradient gr[c][r] and the
// point record (J^-1, w detJ C): F[c][r] = sum_d Ji[3d+r] T[c][d].
__device__ __forceinline__ void point_flux(const float4 r0, const float4 r1, const float4 r2, const float (&gr)[3][3],
                                           float (&F)[3][3]) {
  const float Ji[9] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w, r2.x};
  const float c11 = r2.y, c12 = r2.z, c44 = r2.w;
  float gp[3][3];
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int d = 0; d < 3; ++d)
      gp[c][d] = fmaf(Ji[3 * d], gr[c][0], fmaf(Ji[3 * d + 1], gr[c][1], Ji[3 * d + 2] * gr[c][2]));
  const float exx = gp[0][0], eyy = gp[1][1], ezz = gp[2][2];
  float T[3][3];
  T[0][0] = fmaf(c11, exx, c12 * (eyy + ezz));
  T[1][1] = fmaf(c11, eyy, c12 * (exx + ezz));
  T[2][2] = fmaf(c11, ezz, c12 * (exx + eyy));
  T[0][1] = T[1][0] = c44 * (gp[0][1] + gp[1][0]);
  T[1][2] = T[2][1] = c44 * (gp[1][2] + gp[2][1]);
  T[0][2] = T[2][0] = c44 * (gp[0][2] + gp[2][0]);
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int r = 0; r < 3; ++r) F[c][r] = fmaf(Ji[r], T[c][0], fmaf(Ji[3 + r], T[c][1], Ji[6 + r] * T[c][2]));
}

template <int KR>
struct Shape {
  static constexpr int EPG = 32 / KR;                 // elements per group of three warps
  static constexpr int NG = 4;                        // groups per block, one block per SM (168 registers; five spill)
  static constexpr int NT = NG * 96;
  static constexpr int PV = KR < 4 ? KR : 4;          // columns per staged piece
  static constexpr int PIECES = EPG * NEDOF * (KR / PV);
  static constexpr int PPT = (PIECES + 95) / 96;      // pieces per thread
  static constexpr int UF = EPG * NEDOF * KR;         // p, and zeta fluxes, of a group
  static constexpr int RF = EPG * NGLL * MF_REC;      // point records of a group
  static constexpr int XF = EPG * (NEDOF + NGLL);     // dof numbers, gather positions
  static constexpr int GROUP_F = 2 * UF + 2 * RF + 2 * XF;
  static constexpr size_t SMEM = (size_t)NG * GROUP_F * sizeof(float);
  static_assert(RF % 4 == 0 && UF % 4 == 0 && (2 * XF) % 4 == 0, "16-byte regions");
};

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
}
__device__ __forceinline__ void group_sync(int g) { asm volatile("bar.sync %0, 96;" ::"r"(1 + g) : "memory"); }

template <int KR, bool COMBINE>
__global__ void __launch_bounds__(Shape<KR>::NT, 1) k_apply_mf_planes(
    const float* __restrict__ rec, const int* __restrict__ ge, int nelmt, const float* __restrict__ pold,
    const float* __restrict__ z, float* __restrict__ Y, const ColState* __restrict__ cs,
    const PcgGlobal* __restrict__ G, const int* __restrict__ pos) {
  using S = Shape<KR>;
  constexpr int PV = S::PV, QPD = KR / PV;
  chain_wait();
  if (G && G->all_done) return;
  extern __shared__ __align__(16) float smem[];
  const int grp = threadIdx.x / 96, t = threadIdx.x - 96 * grp, kz = t >> 5, lane = t & 31;
  const int el = lane / KR, j = lane % KR;
  float* U = smem + (size_t)grp * S::GROUP_F;
  float* Fz = U + S::UF;
  float* R = Fz + S::UF;                       // two buffers of records
  int* X = reinterpret_cast<int*>(R + 2 * S::RF);   // two buffers of maps
  const int ngroups = (nelmt + S::EPG - 1) / S::EPG;
  float beta[PV];
#pragma unroll
  for (int k = 0; k < PV; ++k) beta[k] = COMBINE ? (float)cs[PV * (t % QPD) + k].beta : 0.f;   // 96 % QPD == 0
  const float cz0 = kz == 0 ? Dm(0, 0) : kz == 1 ? Dm(1, 0) : Dm(2, 0);
  const float cz1 = kz == 0 ? Dm(0, 1) : kz == 1 ? Dm(1, 1) : Dm(2, 1);
  const float cz2 = kz == 0 ? Dm(0, 2) : kz == 1 ? Dm(1, 2) : Dm(2, 2);
  const float dz0 = kz == 0 ? Dm(0, 0) : kz == 1 ? Dm(0, 1) : Dm(0, 2);   // column kz of D
  const float dz1 = kz == 0 ? Dm(1, 0) : kz == 1 ? Dm(1, 1) : Dm(1, 2);
  const float dz2 = kz == 0 ? Dm(2, 0) : kz == 1 ? Dm(2, 1) : Dm(2, 2);

  // maps and records of group g into buffer b; elements past the end get the
  // sink dof and no position
  auto fetch = [&](int g, int b) {
    const int e0 = g * S::EPG, nv = min(S::EPG, nelmt - e0);
    int* x = X + b * S::XF;
    for (int i = t; i < S::EPG * NEDOF; i += 96) {
      if (i < nv * NEDOF) cp_async4(x + i, ge + (size_t)e0 * NEDOF + i);
      else x[i] = 0;
    }
    for (int i = t; i < S::EPG * NGLL; i += 96) {
      if (i < nv * NGLL) cp_async4(x + S::EPG * NEDOF + i, pos + (size_t)e0 * NGLL + i);
      else x[S::EPG * NEDOF + i] = -1;
    }
    for (int i = t; i < nv * (NGLL * MF_REC / 4); i += 96)
      cp_async16(R + b * S::RF + 4 * i, rec + (size_t)e0 * NGLL * MF_REC + 4 * i);
  };
  // p = beta p_old + z of a group's dof rows, loads first
  float pv[S::PPT][PV], zv[S::PPT][PV];
  auto ask = [&](int b) {
    const int* x = X + b * S::XF;
#pragma unroll
    for (int i = 0; i < S::PPT; ++i) {
      const int q = t + 96 * i;
      if (q < S::PIECES) {
        const size_t o = (size_t)x[q / QPD] * KR + PV * (q % QPD);
        if constexpr (PV == 4) {
          const float4 a = *reinterpret_cast<const float4*>(pold + o);
          pv[i][0] = a.x; pv[i][1] = a.y; pv[i][2] = a.z; pv[i][3] = a.w;
          if (COMBINE) {
            const float4 c = *reinterpret_cast<const float4*>(z + o);
            zv[i][0] = c.x; zv[i][1] = c.y; zv[i][2] = c.z; zv[i][3] = c.w;
          }
        } else {
#pragma unroll
          for (int k = 0; k < PV; ++k) {
            pv[i][k] = pold[o + k];
            if (COMBINE) zv[i][k] = z[o + k];
          }
        }
      }
    }
  };
  auto stage = [&]() {
#pragma unroll
    for (int i = 0; i < S::PPT; ++i) {
      const int q = t + 96 * i;
      if (q < S::PIECES) {
#pragma unroll
        for (int k = 0; k < PV; ++k)
          if (COMBINE) pv[i][k] = fmaf(beta[k], pv[i][k], zv[i][k]);
        if constexpr (PV == 4) {
          *reinterpret_cast<float4*>(U + 4 * q) = make_float4(pv[i][0], pv[i][1], pv[i][2], pv[i][3]);
        } else {
#pragma unroll
          for (int k = 0; k < PV; ++k) U[PV * q + k] = pv[i][k];
        }
      }
    }
  };

  int g = blockIdx.x * S::NG + grp;
  if (g >= ngroups) return;   // whole groups leave: their barriers are their own
  int gstep = gridDim.x * S::NG;
  if (pass_down(G, 0)) { g = ngroups - 1 - g; gstep = -gstep; }
  fetch(g, 0);
  cp_async_wait();
  group_sync(grp);
  ask(0);
  stage();
  for (int b = 0;; b ^= 1) {
    const int gn = g + gstep;
    const bool more = (unsigned)gn < (unsigned)ngroups;
    group_sync(grp);   // p of this group is staged; the other buffer's last readers are done
    if (more) fetch(gn, b ^ 1);
    const float* ue = U + (size_t)el * NEDOF * KR + j;
    float* fe = Fz + (size_t)el * NEDOF * KR + j;
    const float4* Rp = reinterpret_cast<const float4*>(R + b * S::RF) + (el * NGLL + 9 * kz) * 3;
    float u[9][3], y[9][3], fy[9][3];
#pragma unroll
    for (int n = 0; n < 9; ++n)
#pragma unroll
      for (int c = 0; c < 3; ++c) u[n][c] = ue[(3 * (9 * kz + n) + c) * KR];
#pragma unroll
    for (int iy = 0; iy < 3; ++iy) {
      float fx[3][3];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const int n = 3 * iy + i;
        float gr[3][3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          float sx = Dm(i, 0) * u[3 * iy][c];
          if (i != 1) sx = fmaf(Dm(i, 1), u[3 * iy + 1][c], sx);
          gr[c][0] = fmaf(Dm(i, 2), u[3 * iy + 2][c], sx);
          float sy = Dm(iy, 0) * u[i][c];
          if (iy != 1) sy = fmaf(Dm(iy, 1), u[i + 3][c], sy);
          gr[c][1] = fmaf(Dm(iy, 2), u[i + 6][c], sy);
          const float* uz = ue + (3 * n + c) * KR;
          gr[c][2] = fmaf(cz2, uz[54 * KR], fmaf(cz1, uz[27 * KR], cz0 * uz[0]));
        }
        float F[3][3];
        point_flux(Rp[3 * n], Rp[3 * n + 1], Rp[3 * n + 2], gr, F);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          fx[i][c] = F[c][0];
          fy[n][c] = F[c][1];
          fe[(3 * (9 * kz + n) + c) * KR] = F[c][2];
        }
      }
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          float a = Dm(0, i) * fx[0][c];
          if (i != 1) a = fmaf(Dm(1, i), fx[1][c], a);
          y[3 * iy + i][c] = fmaf(Dm(2, i), fx[2][c], a);
        }
    }
#pragma unroll
    for (int iy = 0; iy < 3; ++iy)
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          float a = fmaf(Dm(0, iy), fy[i][c], y[3 * iy + i][c]);
          if (iy != 1) a = fmaf(Dm(1, iy), fy[i + 3][c], a);
          y[3 * iy + i][c] = fmaf(Dm(2, iy), fy[i + 6][c], a);
        }
    cp_async_wait();
    group_sync(grp);   // zeta fluxes stored, p no longer read, the next maps there
    if (more) ask(b ^ 1);
    const int* q = X + b * S::XF + S::EPG * NEDOF + el * NGLL + 9 * kz;
#pragma unroll
    for (int n = 0; n < 9; ++n) {
      const int qn = q[n];
      float* dst = Y + (size_t)qn * 3 * KR + j;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float* f = fe + (3 * n + c) * KR;
        const float a = fmaf(dz2, f[54 * KR], fmaf(dz1, f[27 * KR], fmaf(dz0, f[0], y[n][c])));
        if (qn >= 0) dst[c * KR] = a;
      }
    }
    if (!more) break;
    stage();
    g = gn;
  }
}

// Line form of the same operator, for one and two trials, where a group's
// records would leave room for one or two groups per SM: thread (element,
// xi-line (iy, iz), trial j) owns the line's three nodes and GLL points, the eta
// and zeta terms go through shared memory.  Same arithmetic, same order.
template <int KR>
struct LShape {
  static constexpr int TPE = 9 * KR;                          // threads per element
  static constexpr int EPC = TPE >= 224 ? 1 : 224 / TPE;      // elements per CTA
  static constexpr int NT = ((EPC * TPE + 31) / 32) * 32;
  static constexpr int UF = NEDOF * KR;                       // p per element [node][c][j]
  static constexpr int SF = NGLL * 6 * KR;                    // eta, zeta fluxes [point][c][2][j]
};

template <int KR>
__global__ void __launch_bounds__(LShape<KR>::NT, 2) k_apply_mf_lines(
    const float* __restrict__ rec, const int* __restrict__ ge, int nelmt, const float* __restrict__ pold,
    const float* __restrict__ z, int combine, float* __restrict__ Y, const ColState* __restrict__ cs,
    const PcgGlobal* __restrict__ G, const int* __restrict__ pos) {
  using S = LShape<KR>;
  if (G && G->all_done) return;
  __shared__ __align__(16) float sU[S::EPC][S::UF];
  __shared__ __align__(16) float sS[S::EPC][S::SF];
  const int t = threadIdx.x;
  const int el = t / S::TPE, rem = t - el * S::TPE;
  const int line = rem / KR, j = rem - line * KR;
  const int iy = line % 3, iz = line / 3;
  const int nbase = 3 * iy + 9 * iz;  // node ix = 0 of the line
  const bool act = el < S::EPC;
  const float beta = (act && combine) ? (float)cs[j].beta : 0.f;
  float* U = sU[act ? el : 0];
  float* Fs = sS[act ? el : 0];
  const int estride = gridDim.x * S::EPC;
  int e = blockIdx.x * S::EPC + el;
  // software pipeline: next element's dof numbers during the
  // first phase, its p and z rows during the second
  int gd[9];
  float pv[9], zv[9];
  auto load_dofs = [&](int ee, int (&g)[9]) {
#pragma unroll
    for (int k = 0; k < 9; ++k)
      g[k] = (act && ee < nelmt) ? __ldg(ge + (size_t)ee * NEDOF + 3 * nbase + k) : 0;
  };
  auto load_p = [&](const int (&g)[9]) {
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      pv[k] = pold[(size_t)g[k] * KR + j];
      zv[k] = combine ? z[(size_t)g[k] * KR + j] : 0.f;
    }
  };
  load_dofs(e, gd);
  load_p(gd);
  for (int e0 = blockIdx.x * S::EPC; e0 < nelmt; e0 += estride, e += estride) {
    const bool valid = act && e < nelmt;
    float uR[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float u = valid ? (combine ? fmaf(beta, pv[3 * i + c], zv[3 * i + c]) : pv[3 * i + c]) : 0.f;
        uR[i][c] = u;
        if (act) U[(3 * (nbase + i) + c) * KR + j] = u;
      }
    int gdn[9];
    load_dofs(e + estride, gdn);
    __syncthreads();
    float Fx[3][3];  // xi fluxes of the line's points [i][c]
    if (valid) {
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const int q = nbase + i;
        const float4* R = reinterpret_cast<const float4*>(rec + ((size_t)e * NGLL + q) * MF_REC);
        const float4 r0 = __ldg(R), r1 = __ldg(R + 1), r2 = __ldg(R + 2);
        float gr[3][3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          float sx = 0.f, sy = 0.f, sz = 0.f;
#pragma unroll
          for (int tt = 0; tt < 3; ++tt) {
            sx = fmaf(Dm(i, tt), uR[tt][c], sx);
            sy = fmaf(Dm(iy, tt), U[(3 * (i + 3 * tt + 9 * iz) + c) * KR + j], sy);
            sz = fmaf(Dm(iz, tt), U[(3 * (i + 3 * iy + 9 * tt) + c) * KR + j], sz);
          }
          gr[c][0] = sx;
          gr[c][1] = sy;
          gr[c][2] = sz;
        }
        float F[3][3];
        point_flux(r0, r1, r2, gr, F);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          Fx[i][c] = F[c][0];
          Fs[((3 * q + c) * 2 + 0) * KR + j] = F[c][1];
          Fs[((3 * q + c) * 2 + 1) * KR + j] = F[c][2];
        }
      }
    }
    load_p(gdn);
    __syncthreads();
    if (valid) {
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const int n = nbase + i;
        float y[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          float acc = 0.f;
#pragma unroll
          for (int tt = 0; tt < 3; ++tt) acc = fmaf(Dm(tt, i), Fx[tt][c], acc);
#pragma unroll
          for (int tt = 0; tt < 3; ++tt) acc = fmaf(Dm(tt, iy), Fs[((3 * (i + 3 * tt + 9 * iz) + c) * 2 + 0) * KR + j], acc);
#pragma unroll
          for (int tt = 0; tt < 3; ++tt) acc = fmaf(Dm(tt, iz), Fs[((3 * (i + 3 * iy + 9 * tt) + c) * 2 + 1) * KR + j], acc);
          y[c] = acc;
        }
        const int q = __ldg(pos + (size_t)e * NGLL + n);
        if (q >= 0) {
          float* dst = Y + (size_t)q * 3 * KR + j;
          dst[0] = y[0];
          dst[KR] = y[1];
          dst[2 * KR] = y[2];
        }
      }
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) gd[k] = gdn[k];
    __syncthreads();
  }
}

// Record of GLL point q of operator element le (element elist[le]):
// J^-1 (row-major, as cached by the geometry kernel) and the compute_cmat
// constants times w_q detJ_q, rounded to FP32.
__global__ void k_mf_record(const double* __restrict__ geo, const int* __restrict__ mat_id,
                            const int* __restrict__ elist, int nel, const double* __restrict__ ym,
                            const double* __restrict__ nu, float* __restrict__ rec) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= nel * NGLL) return;
  const int le = tid / NGLL, q = tid - le * NGLL;
  const int e = elist ? elist[le] : le;
  const int im = mat_id[e] - 1;
  const double E = ym[im], v = nu[im];
  const double onepv = 1.0 + v, onemv = 1.0 - v, onem2v = 1.0 - 2.0 * v;
  const double Ef = E / (onepv * onem2v);
  const double w1[3] = {1.0 / 3.0, 4.0 / 3.0, 1.0 / 3.0};
  const double* g = geo + ((size_t)e * NGLL + q) * GEO_STRIDE;
  const double wd = w1[q % 3] * w1[(q / 3) % 3] * w1[q / 9] * g[9];
  float* r = rec + ((size_t)le * NGLL + q) * MF_REC;
#pragma unroll
  for (int i = 0; i < 9; ++i) r[i] = (float)g[i];
  r[9] = (float)(wd * onemv * Ef);
  r[10] = (float)(wd * v * Ef);
  r[11] = (float)(wd * 0.5 * onem2v * Ef);
}

}  // namespace mf

template <int KR>
void launch_apply_mf(const float* rec, const int* ge, int nelmt, const float* pold, const float* z, int combine,
                     float* Y, const ColState* cs, const PcgGlobal* G, const int* pos, cudaStream_t s) {
  if constexpr (KR < 4) {
    using S = mf::LShape<KR>;
    const int nb = (nelmt + S::EPC - 1) / S::EPC;
    const int grid = nb < 152 * 8 ? nb : 152 * 8;
    if (grid < 1) return;
    mf::k_apply_mf_lines<KR><<<grid, S::NT, 0, s>>>(rec, ge, nelmt, pold, z, combine, Y, cs, G, pos);
  } else {
    using S = mf::Shape<KR>;
    static std::atomic<unsigned long long> plain{}, combined{};
    if (combine) allow_smem(combined, (const void*)mf::k_apply_mf_planes<KR, true>, S::SMEM);
    else allow_smem(plain, (const void*)mf::k_apply_mf_planes<KR, false>, S::SMEM);
    const int ng = (nelmt + S::EPG - 1) / S::EPG, nb = (ng + S::NG - 1) / S::NG;
    const int grid = nb < 152 ? nb : 152;
    if (grid < 1) return;
    launch_chained(combine ? mf::k_apply_mf_planes<KR, true> : mf::k_apply_mf_planes<KR, false>, grid, S::NT, S::SMEM, s,
                   rec, ge, nelmt, pold, z, Y, cs, G, pos);
  }
}

void launch_mf_record(const double* geo, const int* mat_id, const int* elist, int nel, const double* ym,
                      const double* nu, float* rec, cudaStream_t s) {
  if (nel <= 0 || !rec) return;
  const int n = nel * NGLL;
  mf::k_mf_record<<<(n + 255) / 256, 256, 0, s>>>(geo, mat_id, elist, nel, ym, nu, rec);
}

template void launch_apply_mf<1>(const float*, const int*, int, const float*, const float*, int, float*,
                                 const ColState*, const PcgGlobal*, const int*, cudaStream_t);
template void launch_apply_mf<2>(const float*, const int*, int, const float*, const float*, int, float*,
                                 const ColState*, const PcgGlobal*, const int*, cudaStream_t);
template void launch_apply_mf<4>(const float*, const int*, int, const float*, const float*, int, float*,
                                 const ColState*, const PcgGlobal*, const int*, cudaStream_t);
template void launch_apply_mf<8>(const float*, const int*, int, const float*, const float*, int, float*,
                                 const ColState*, const PcgGlobal*, const int*, cudaStream_t);
template void launch_apply_mf<16>(const float*, const int*, int, const float*, const float*, int, float*,
                                  const ColState*, const PcgGlobal*, const int*, cudaStream_t);

}  // namespace sg
