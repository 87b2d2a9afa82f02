// sg_pcg_persist64.cu -- the FP64 PCG iterations (one right-hand side) as one
// persistent cooperative kernel, for the model's stored sparse matrices and
// for the drop-in's dense ones.
//
// What bounds it: the FP64 unit takes a warp instruction in some 19 cycles, so
// the element products (171 fused multiply-adds a lane with lane = node and 27
// of 32 lanes at work) are nearly all of an iteration from a few thousand
// elements on, and below that the launches, tails and round trips of three
// kernels are.  So
//   * a lane is one row of an element's product and the rows of a block's
//     elements are cut into warps without regard to element borders: no lane
//     idles (144 FP64 instructions an element instead of 171, or of the 243 of
//     a dense column sweep);
//   * only the 57 columns a row can be coupled to are multiplied.  The
//     drop-in's dense matrices are checked for that pattern on the device once
//     per call (k_pack_rows) and packed; matrices that do not have it take the
//     dense kernel;
//   * a block's matrices stay in shared memory for the whole launch while they
//     fit, else they stream through two buffers filled by bulk copies, the
//     next iteration's first group on its way during the vector phases;
//   * the vector phases hand out warps, not blocks: the reference order of the
//     dots groups 32 threads first, so each such warp may run on any SM, and
//     a small mesh's few blocks of them do not queue on few FP64 units;
//   * maxima are taken on the bits of the absolute values (integer unit), and
//     the stop test divides only when the products do not decide it;
//   * the phases of an iteration are separated by the counter barrier of
//     sg_pcg_persist.cu.
//
// The arithmetic and its order are those of k_apply_dense64 / k_apply_sparse*,
// k_pcg_gather and k_pcg_update: products in column order (an exact zero adds
// nothing), slots in element order, and dots over the same virtual grid of
// 256-thread blocks with the same trees, so a solve is bitwise the one of the
// separate kernels.
//
// us per iteration, separate kernels (with short tails) -> this: 300 elements
// dense 43 -> 16, sparse 37 -> 16; 12,000 elements sparse 256 -> 158, of which the
// products take 119 (19 cycles for each FP64 warp instruction).  Code that one
// warp runs once per iteration is kept short: unrolled twofold over nodes, the
// gather took 10 us instead of 4.
//
// Every wait is bounded; a timeout sets the solve's error word, the block
// waits (bounded) for its own copies and leaves, and the others follow.
#include <cstdint>
#include <cstdlib>
#include <type_traits>

#include "sg_kernels.cuh"

namespace sg {

namespace p64 {

constexpr int NT = 512, NWARP = NT / 32;
constexpr int MAX_BLOCKS = 152;
constexpr int POLL_TRIES = 1 << 20;
constexpr int VT = RED_THREADS;          // threads of a virtual block
constexpr unsigned FULL = 0xffffffffu;

template <bool ROWS>
struct Lay {
  static constexpr int STRIDE = ROWS ? ROW_STRIDE : KS_STRIDE;        // doubles per element
  static constexpr int GE = ROWS ? 2 : 5;                             // elements per streamed group
  static constexpr int RES = ROWS ? 5 : 10;                           // elements that stay in shared memory
  static constexpr int NP = RES > 2 * GE ? RES : 2 * GE;              // direction slots
  static constexpr size_t SMEM = (size_t)NP * (STRIDE + NEDOF) * sizeof(double);
  static_assert(RES <= NP && 2 * GE <= NP && GE * NEDOF <= NT, "buffers");
  static_assert((STRIDE * sizeof(double)) % 16 == 0, "bulk copies");
};

struct Args {
  const double* K;
  const int *ge, *pos, *nbr;
  int nelmt;
  const int *gptr, *gdof;
  int ngroups, n1, ggrid, ugrid;         // virtual grids of the gather and the update
  double *u, *r, *z, *p, *kp, *Y;
  const double* dp;
  ColState* cs;
  PcgGlobal* G;
  double* part;                          // warp partials: p.kp [8 ggrid], r.z, max|p|, max|u| [8 ugrid] each
  unsigned* count;
  int chunk;
};

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity) {
  for (int tries = 0; tries < (1 << 22); ++tries) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}
// |x| as an integer that orders like it; a NaN counts as 0, as fmax has it
__device__ __forceinline__ unsigned long long mag(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
  return b > 0x7ff0000000000000ull ? 0ull : b;
}
__device__ __forceinline__ unsigned long long warp_max(unsigned long long x) {
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    const unsigned long long y = __shfl_xor_sync(FULL, x, o);
    x = x > y ? x : y;
  }
  return x;
}
// 0 + x[0] + x[1] + ... + x[n - 1], one add after the other, loads ahead of them
__device__ __forceinline__ double chain(const double* x, int n) {
  double s = 0.0;
  int i = 0;
#pragma unroll 1
  for (; i + 8 <= n; i += 8) {
    double v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = x[i + k];
#pragma unroll
    for (int k = 0; k < 8; ++k) s += v[k];
  }
#pragma unroll 1
  for (; i < n; ++i) s += x[i];
  return s;
}
// a block's sum from its eight warps' partials
__device__ __forceinline__ double block_partial(const double* part, int vb) {
  const double2* w = reinterpret_cast<const double2*>(part + (size_t)vb * (VT / 32));
  double2 x[VT / 64];
#pragma unroll
  for (int i = 0; i < VT / 64; ++i) x[i] = __ldcg(w + i);
  double v = 0.0;
#pragma unroll
  for (int i = 0; i < VT / 64; ++i) { v += x[i].x; v += x[i].y; }
  return v;
}

// Rows [r0, r1) of the elements from efirst on, whose matrices start at kb and
// directions at ps.
template <bool ROWS>
__device__ __forceinline__ void row_products(const Args& A, const double* kb, const double* ps, int efirst, int r0,
                                             int r1, const int* nbr, int warp, int lane) {
  using L = Lay<ROWS>;
  for (int row = r0 + warp * 32 + lane; row < r1; row += NT) {
    const int el = row / NEDOF, rr = row - el * NEDOF, n = rr / 3, cc = rr - 3 * n;
    const double* k = kb + (size_t)el * L::STRIDE;
    const double* pe = ps + el * NEDOF;
    const int* tb = nbr + n * KS_NBR;
    double y = 0.0;
#pragma unroll
    for (int s = 0; s < KS_NBR; ++s) {
      const int pk = tb[s], m = pk & 31;
      if constexpr (ROWS) {
#pragma unroll
        for (int d = 0; d < 3; ++d) y = fma(k[(3 * s + d) * NEDOF + rr], pe[3 * m + d], y);
      } else {
        // stored (n, m) row-major, or (m, n) read transposed
        const bool tr = ((pk >> 5) & 3) == 2;
        const double* kk = k + (pk >> 8) + (tr ? cc : 3 * cc);
        const int sd = tr ? 3 : 1;
#pragma unroll
        for (int d = 0; d < 3; ++d) y = fma(kk[d * sd], pe[3 * m + d], y);
      }
    }
    const int q = __ldg(A.pos + (size_t)(efirst + el) * NGLL + n);
    if (q >= 0) A.Y[(size_t)q * 3 + cc] = y;
  }
}

template <bool ROWS>
__global__ void __launch_bounds__(NT, 1) k_pcg_persistent64(Args A) {
  using L = Lay<ROWS>;
  extern __shared__ __align__(128) double dsm[];
  double* kb = dsm;                                   // matrices: resident, or two groups
  double* ps = dsm + (size_t)L::NP * L::STRIDE;       // directions of the same elements
  __shared__ int nbr[NGLL * KS_NBR];
  __shared__ __align__(8) uint64_t bar[2];
  __shared__ double spart[NPART], sfin[VT];
  __shared__ int4 smap[NWARP][2][32];
  __shared__ int smap2[NWARP][2][32];
  __shared__ unsigned long long smax[NWARP][2];
  __shared__ double s_alpha, s_beta, s_rz, s_maxp, s_maxu;
  __shared__ int s_done, s_failed;
  PcgGlobal* G = A.G;
  if (G->all_done) return;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int grid = gridDim.x, bid = blockIdx.x;
  const double tol = A.cs[0].tol;
  if (t == 0) {
    s_rz = A.cs[0].rz; s_alpha = A.cs[0].alpha; s_beta = A.cs[0].beta;
    s_maxp = A.cs[0].maxp; s_maxu = A.cs[0].maxu; s_done = 0; s_failed = 0;
    for (int b = 0; b < 2; ++b)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar + b)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = t; i < NGLL * KS_NBR; i += NT) nbr[i] = A.nbr[i];
  int it = G->it;
  const int maxiter = G->maxiter;
  unsigned arrivals = 0;
  // the block's rows: whole warps of 32 while the matrices they touch stay in
  // shared memory, else whole elements
  const int rows = A.nelmt * NEDOF, nchunk = (rows + 31) / 32, rper = (nchunk + grid - 1) / grid * 32;
  const bool resident = (rper + NEDOF - 2) / NEDOF + 1 <= L::RES;   // a run of rper rows meets no more elements
  const int per = (A.nelmt + grid - 1) / grid;
  const int r0 = resident ? min(rows, bid * rper) : min(A.nelmt, bid * per) * NEDOF;
  const int r1 = resident ? min(rows, r0 + rper) : min(A.nelmt, bid * per + per) * NEDOF;
  const int e0 = min(r0 / NEDOF, A.nelmt), nel = r1 > r0 ? (r1 - 1) / NEDOF + 1 - e0 : 0;
  const int ngrp = (nel + L::GE - 1) / L::GE;
  unsigned uses = 0;        // groups copied so far (buffer uses % 2), the same in all threads
  unsigned waited = 0;
  __syncthreads();
  auto copy_group = [&](int g) {
    if (t == 0) {
      const int first = g * L::GE, n = min(L::GE, nel - first);
      const unsigned b = uses & 1, bytes = (unsigned)n * L::STRIDE * 8;
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar + b)), "r"(bytes)
                   : "memory");
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
              smem_u32(kb + (size_t)b * L::GE * L::STRIDE)),
          "l"(A.K + (size_t)(e0 + first) * L::STRIDE), "r"(bytes), "r"(smem_u32(bar + b))
          : "memory");
    }
    ++uses;
  };
  if (resident) {
    const double2* src = reinterpret_cast<const double2*>(A.K + (size_t)e0 * L::STRIDE);
    for (int i = t; i < nel * (L::STRIDE / 2); i += NT) reinterpret_cast<double2*>(kb)[i] = __ldcs(src + i);
  } else if (nel > 0) {
    copy_group(0);
  }
  auto barrier = [&]() -> bool {
    __syncthreads();
    bool good = true;
    if (t == 0) {
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(A.count) : "memory");
      arrivals += (unsigned)grid;
      unsigned n;
      int tries = 0;
      do {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(n) : "l"(A.count) : "memory");
        if (++tries > POLL_TRIES) good = false;
      } while (n < arrivals && good);
      if (!good) atomicExch(&G->err, 1);
    }
    return !__syncthreads_or(!good);
  };
  // direction value i of the elements from first on
  auto direction = [&](int first, int i) -> double {
    const int gd = __ldg(A.ge + (size_t)(e0 + first) * NEDOF + i);
    return fma(s_beta, __ldcg(A.p + gd), __ldcg(A.z + gd));
  };
  // slot range and dof numbers of node g, {a, b, dof 0, dof 1} and dof 2
  auto load_map = [&](int g, int4& m, int& gd2) {
    m = make_int4(0, 0, 0, 0);
    gd2 = 0;
    if (g < A.ngroups) {
      m = make_int4(__ldg(A.gptr + g), __ldg(A.gptr + g + 1), __ldg(A.gdof + 3 * g), __ldg(A.gdof + 3 * g + 1));
      gd2 = __ldg(A.gdof + 3 * g + 2);
    }
  };
  for (int j = 0; j < 2; ++j) {
    int4 m;
    int gd2;
    load_map((bid + warp * grid) * 32 + lane + j * A.ggrid * VT, m, gd2);
    smap[warp][j][lane] = m;
    smap2[warp][j][lane] = gd2;
  }
  double* partB = A.part;
  constexpr int VW = VT / 32;
  double* partZ = A.part + VW * A.ggrid;
  unsigned long long* partP = reinterpret_cast<unsigned long long*>(partZ + VW * A.ugrid);
  unsigned long long* partU = partP + VW * A.ugrid;
  bool ok = true;
  for (int k = 0; k < A.chunk && ok; ++k) {
    // ---- element products of p = z + beta p_old ----
    if (resident) {
      for (int i = t; i < nel * NEDOF; i += NT) ps[i] = direction(0, i);
      __syncthreads();
      row_products<ROWS>(A, kb, ps, e0, r0 - e0 * NEDOF, r1 - e0 * NEDOF, nbr, warp, lane);
    } else {
      if (t < min(L::GE, nel) * NEDOF) ps[t] = direction(0, t);
      for (int g = 0; g < ngrp; ++g) {
        const int b = waited & 1, n = min(L::GE, nel - g * L::GE), nn = min(L::GE, nel - (g + 1) * L::GE);
        // the next group, or the next iteration's first, while this one is computed
        copy_group(g + 1 < ngrp ? g + 1 : 0);
        double nd = 0.0;
        if (t < nn * NEDOF) nd = direction((g + 1) * L::GE, t);
        ok = mbar_wait(bar + b, (waited >> 1) & 1);
        if (__syncthreads_or(!ok)) { ok = false; break; }
        ++waited;
        row_products<ROWS>(A, kb + (size_t)b * L::GE * L::STRIDE, ps + (g & 1) * L::GE * NEDOF, e0 + g * L::GE, 0,
                           n * NEDOF, nbr, warp, lane);
        if (t < nn * NEDOF) ps[((g + 1) & 1) * L::GE * NEDOF + t] = nd;
        __syncthreads();
      }
      if (!ok) {
        if (t == 0) atomicExch(&G->err, 1);
        break;
      }
    }
    if (!barrier()) { ok = false; break; }
    // ---- kp, p and p.kp: warp w of the gather's grid takes 32 nodes, then the
    // 32 a grid further on, ... ----
    const double beta = s_beta;
    for (int w = bid + warp * grid; w < VW * A.ggrid; w += NWARP * grid) {
      double dot = 0.0;
      const int gs = A.ggrid * VT;
      const bool mapped = w == bid + warp * grid;   // the first such warp keeps two nodes' maps in shared memory
#pragma unroll 1
      for (int j = 0; w * 32 + j * gs < A.ngroups; ++j) {
        int4 m;
        int gd2;
        if (mapped && j < 2) {
          m = smap[warp][j][lane];
          gd2 = smap2[warp][j][lane];
        } else {
          load_map(w * 32 + lane + j * gs, m, gd2);
        }
        const int gd[3] = {m.z, m.w, gd2};
        double pv[3], zv[3], y[4][3], acc[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          pv[d] = __ldcg(A.p + gd[d]);
          zv[d] = __ldcg(A.z + gd[d]);
        }
        // absent slots add +0, which changes no sum that began at +0
        int s0 = m.x;
#pragma unroll 1
        do {
          const double* yp = A.Y + (size_t)s0 * 3;
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int d = 0; d < 3; ++d) y[i][d] = s0 + i < m.y ? __ldcg(yp + 3 * i + d) : 0.0;
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int d = 0; d < 3; ++d) acc[d] = acc[d] + y[i][d];
          s0 += 4;
        } while (s0 < m.y);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          if (!gd[d]) continue;
          const double pn = fma(beta, pv[d], zv[d]);
          dot = fma(pn, acc[d], dot);
          A.p[gd[d]] = pn;
          A.kp[gd[d]] = acc[d];
        }
      }
#pragma unroll
      for (int o = 16; o >= 1; o >>= 1) dot += __shfl_xor_sync(FULL, dot, o);
      if (lane == 0) __stcg(partB + w, dot);
    }
    if (!barrier()) { ok = false; break; }
    // alpha: the partials in the order of the last block's sum
    for (int b = t; b < A.ggrid; b += NT) spart[b] = block_partial(partB, b);
    __syncthreads();
    if (t < VT) {
      double v = 0.0;
      for (int b = t; b < A.ggrid; b += VT) v += spart[b];
      sfin[t] = v;
    }
    __syncthreads();
    if (t == 0) s_alpha = s_rz / chain(sfin, min(VT, A.ggrid));
    __syncthreads();
    // ---- u, r, z, max-norms and r.z, by warps of the update's grid ----
    const double alpha = s_alpha;
    for (int w = bid + warp * grid; w < VW * A.ugrid; w += NWARP * grid) {
      unsigned long long mp = 0, mu = 0;
      double rz = 0.0;
      const size_t stride = (size_t)A.ugrid * VT;
      for (size_t i0 = (size_t)w * 32 + lane; i0 < (size_t)A.n1; i0 += 4 * stride) {
        double pv[4], uv[4], rv[4], kv[4], dv[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const size_t i = i0 + q * stride;
          if (i < (size_t)A.n1) {
            pv[q] = __ldcg(A.p + i); uv[q] = __ldcg(A.u + i); rv[q] = __ldcg(A.r + i); kv[q] = __ldcg(A.kp + i);
            dv[q] = __ldg(A.dp + i);
          }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const size_t i = i0 + q * stride;
          if (i >= (size_t)A.n1) continue;
          const double un = fma(alpha, pv[q], uv[q]), rn = fma(-alpha, kv[q], rv[q]), zn = dv[q] * rn;
          A.u[i] = un; A.r[i] = rn; A.z[i] = zn;
          mp = max(mp, mag(pv[q]));
          mu = max(mu, mag(un));
          rz = fma(rn, zn, rz);
        }
      }
      mp = warp_max(mp);
      mu = warp_max(mu);
#pragma unroll
      for (int o = 16; o >= 1; o >>= 1) rz = rz + __shfl_xor_sync(FULL, rz, o);
      if (lane == 0) { __stcg(partZ + w, rz); __stcg(partP + w, mp); __stcg(partU + w, mu); }
    }
    if (!barrier()) { ok = false; break; }
    // stop test and beta, identical in every block: r.z over interleaved
    // 64-block strides as the last block of k_pcg_update sums it
    ++it;
    {
      constexpr int NJ = VT / 4;
      for (int b = t; b < A.ugrid; b += NT) spart[b] = block_partial(partZ, b);
      unsigned long long mp = 0, mu = 0;
      for (int w = t; w < VW * A.ugrid; w += NT) {
        mp = max(mp, __ldcg(partP + w));
        mu = max(mu, __ldcg(partU + w));
      }
      mp = warp_max(mp);
      mu = warp_max(mu);
      if (lane == 0) { smax[warp][0] = mp; smax[warp][1] = mu; }
      __syncthreads();
      if (t < NJ) {
        double v = 0.0;
        for (int b = t; b < A.ugrid; b += NJ) v += spart[b];
        sfin[t] = v;
      } else if (warp == NWARP - 1) {
        // |alpha| max|p| / max|u| <= tol, divided only where the products are close
        mp = lane < NWARP ? smax[lane][0] : 0;
        mu = lane < NWARP ? smax[lane][1] : 0;
        mp = warp_max(mp);
        mu = warp_max(mu);
        if (lane == 0) {
          const double dp = __longlong_as_double((long long)mp), du = __longlong_as_double((long long)mu);
          const double a = fabs(s_alpha) * dp, b = tol * du, eps = 1e-14 * b;
          s_maxp = dp; s_maxu = du;
          s_done = a < b - eps ? 1 : a > b + eps ? 0 : a / du <= tol;
        }
      }
      __syncthreads();
      if (t == 0) {
        if (!s_done) {
          if (it >= maxiter) {
            s_done = 1; s_failed = 1;
          } else {
            const double s = chain(sfin, min(NJ, A.ugrid));
            s_beta = s / s_rz;
            s_rz = s;
          }
        }
      }
      __syncthreads();
    }
    if (s_done) break;
  }
  // copies still on their way must land before the block leaves (bounded)
  for (; waited < uses; ++waited) mbar_wait(bar + (waited & 1), (waited >> 1) & 1);
  if (!ok) return;
  if (bid == 0 && t == 0) {
    ColState& c = A.cs[0];
    c.rz = s_rz; c.alpha = s_alpha; c.beta = s_beta; c.maxp = s_maxp; c.maxu = s_maxu;
    if (s_done) { c.done = 1; c.failed = s_failed; c.iters = s_failed ? maxiter + 1 : it; }
    G->it = it;
    G->all_done = s_done;
  }
}

// Packs dense column-major 81x81 matrices into [57][81]: entry (3 s + d, row)
// is K(row, 3 m + d) with m the s-th node coupled to the row's node.  *other
// is set when an entry outside that pattern is not zero (or is not a number).
__global__ void __launch_bounds__(256) k_pack_rows(const double* __restrict__ K, const int* __restrict__ nbr_g,
                                                   double* __restrict__ out, int* __restrict__ other) {
  __shared__ signed char slot[NGLL][NGLL];   // s of (n, m), or -1
  for (int i = threadIdx.x; i < NGLL * NGLL; i += blockDim.x) slot[i / NGLL][i % NGLL] = -1;
  __syncthreads();
  for (int i = threadIdx.x; i < NGLL * KS_NBR; i += blockDim.x) slot[i / KS_NBR][nbr_g[i] & 31] = (signed char)(i % KS_NBR);
  __syncthreads();
  const double* k = K + (size_t)blockIdx.x * NEDOF * NEDOF;
  double* o = out + (size_t)blockIdx.x * ROW_STRIDE;
  bool bad = false;
  for (int i = threadIdx.x; i < NEDOF * NEDOF; i += blockDim.x) {
    const int col = i / NEDOF, row = i - col * NEDOF, s = slot[row / 3][col / 3];
    const double v = __ldcs(k + i);
    if (s >= 0) o[(3 * s + col % 3) * NEDOF + row] = v;
    else bad = bad || !(v == 0.0);
  }
  if (threadIdx.x < ROW_STRIDE - 3 * KS_NBR * NEDOF) o[3 * KS_NBR * NEDOF + threadIdx.x] = 0.0;
  if (__syncthreads_or(bad) && threadIdx.x == 0) *other = 1;
}

template <bool ROWS>
static bool launch(Args A, int grid, cudaStream_t s) {
  using L = Lay<ROWS>;
  static std::atomic<unsigned long long> allowed{};
  if (!allow_smem(allowed, (const void*)k_pcg_persistent64<ROWS>, L::SMEM)) {
    cudaGetLastError();
    return false;
  }
  void* args[] = {&A};
  if (cudaLaunchCooperativeKernel((const void*)k_pcg_persistent64<ROWS>, grid, NT, args, L::SMEM, s) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  add_launches(1);
  return true;
}

}  // namespace p64

void launch_pack_rows(const double* K, int nelmt, const int* d_nbr, double* out, int* other, cudaStream_t s) {
  cudaMemsetAsync(other, 0, sizeof(int), s);
  if (nelmt <= 0) return;
  p64::k_pack_rows<<<nelmt, 256, 0, s>>>(K, d_nbr, out, other);
  add_launches(1);
}

// Up to `chunk` PCG iterations (reference step test).  rows: K is packed by
// k_pack_rows, else the sparse symmetric layout.  False when it cannot run.
bool launch_pcg_persistent64(bool rows, const double* K, const int* ge, int nelmt, const int* pos, const int* d_nbr,
                             const GatherTopo& T, int n1, double* u, double* r, double* z, double* p, double* kp,
                             double* Y, const double* dp, ColState* cs, PcgGlobal* G, double* part, int chunk,
                             cudaStream_t s) {
  // the virtual grids are those of k_pcg_gather and k_pcg_update
  auto red = [](size_t items, size_t per) {
    const size_t g = (items + per - 1) / per;
    return (int)(g < 1 ? 1 : g > (size_t)NPART ? (size_t)NPART : g);
  };
  const int ggrid = red(T.ngroups, VGATHER), ugrid = red(n1, VUPDATE);
  long grid = ((long)nelmt * NEDOF + 31) / 32;   // a warp of rows per block, at least
  if (grid < 8L * ugrid) grid = 8L * ugrid;
  if (grid > p64::MAX_BLOCKS) grid = p64::MAX_BLOCKS;
  unsigned* count = reinterpret_cast<unsigned*>(part + RED_THREADS / 32 * (ggrid + 3 * ugrid));
  static_assert(RED_THREADS / 32 * 4 * NPART + 1 <= NPART * 16 * 4, "partials and the count fit the buffer");
  cudaMemsetAsync(count, 0, sizeof(unsigned), s);
  const p64::Args A{K, ge, pos, d_nbr, nelmt, T.d_ptr, T.d_dof, T.ngroups, n1, ggrid, ugrid,
                    u, r, z, p, kp, Y, dp, cs, G, part, count, chunk};
  return rows ? p64::launch<true>(A, (int)grid, s) : p64::launch<false>(A, (int)grid, s);
}

}  // namespace sg
