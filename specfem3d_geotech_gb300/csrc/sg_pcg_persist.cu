// sg_pcg_persist.cu -- the FP32 PCG iterations of small and medium meshes as
// one persistent cooperative kernel.
//
// On a few thousand elements a PCG iteration (element apply, gather, vector
// update) is a microsecond or two of work, but three dependent kernels cost
// some 12 us each: the launch, a chain of L2 round trips (control word,
// column state, data), and a last-block reduction behind an atomic.  Here a
// chunk of iterations runs inside one launch of one block per SM:
//
//   A  element products of p = z + beta p_old -> Y          | barrier
//   B  kp = sum of Y per node, p = z + beta p_old, p.kp      | barrier, sums
//   C  u += alpha p, r -= alpha kp, z = D r, r.z, r.r        | barrier, sums
//
// The barrier is one counter: a block's first thread adds to it with release
// order and alone polls it (2,600 cycles on 152 blocks; flags or partials that
// every block polls from every other took 8,700, clusters with one flag each
// 3,700).  Partial sums are written before the barrier of their phase and
// added by every block after it, in the same order, so all blocks take the
// same decisions and results are deterministic.
//
// FP64 arithmetic is kept out of the loop: the trees over 15 warps and up to 32
// sums took longer than the barrier.  Sums and the scalars formed from them are
// three floats (sg_sum3.cuh), more bits than FP64 keeps, and rounded to FP32 once,
// as the vector operations take them.  Against pairs that costs some 25 cycles an
// addition, of 20 one after the other; on small meshes the nodes are spread over
// all blocks, so that few warps of a block have sums, which gains as much.
//
// A dof row's u, r, p stay in the registers of the thread that owns it while
// the mesh is small enough (R pieces of up to four columns a thread, R = 1 or
// 2, for one or two columns also 4, for one 8); beyond that (R = 0) they stream
// through L2 (5,880 elements and one column: 17.9 us an iteration streamed, 15.2
// in registers).  The element maps and point
// records of a block's elements stay in shared memory where they fit.
//
// Phase A gives a warp one element and up to four columns, lane = node: the
// warp is its own barrier, each lane's four columns are independent chains,
// and all shared traffic is 16 bytes a lane.  The arithmetic per column and its
// order are those of sg_apply_mf.cu, and phases B and C do that of the gather
// and update kernels, so the two ways differ only in how the dots are grouped.
//
// Waits are bounded: a block that polls too long sets the solve's error word
// and leaves, the others' waits then run out as well, the launch ends and the
// solve reports SG_ERR_TIMEOUT without launching another chunk.
#include <cstdint>
#include <cstdlib>
#include <type_traits>

#include "sg_kernels.cuh"
#include "sg_sum3.cuh"

namespace sg {

namespace pp {

constexpr int NT = 480;               // 15 warps; a multiple of 3, 6 and 12 pieces per node
constexpr int NWARP = NT / 32;
constexpr int MAX_BLOCKS = 152;       // one block per SM
constexpr int POLL_TRIES = 1 << 20;   // bounded wait, below a second

__device__ __forceinline__ Sum3 shfl_xor(const Sum3& x, int o) {
  return Sum3{__shfl_xor_sync(0xffffffffu, x.h, o), __shfl_xor_sync(0xffffffffu, x.l, o),
              __shfl_xor_sync(0xffffffffu, x.m, o)};
}

// Sums x[0..N) over the lanes that differ in bits O, O/2, ..., O0, halving the
// values a lane carries at each step while it has several (N - 1 + steps adds
// instead of N * steps): the lane ends with value index() in x[0].
template <int N, int O, int O0>
struct Reduce {
  static __device__ __forceinline__ void run(Sum3 (&x)[N], int lane) {
    if constexpr (O >= O0) {
      if constexpr (N > 1) {
        const bool up = lane & O;
        Sum3 y[N / 2];
#pragma unroll
        for (int i = 0; i < N / 2; ++i) {
          const Sum3 keep = up ? x[i + N / 2] : x[i], send = up ? x[i] : x[i + N / 2];
          y[i] = keep;
          y[i].add(shfl_xor(send, O));
        }
        Reduce<N / 2, O / 2, O0>::run(y, lane);
        x[0] = y[0];
      } else {
        x[0].add(shfl_xor(x[0], O));
        Reduce<N, O / 2, O0>::run(x, lane);
      }
    }
  }
};

// VW consecutive floats; loads go through L2 (other blocks write the data)
template <int VW>
struct Vec {
  float v[VW];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int k = 0; k < VW; ++k) v[k] = 0.f;
  }
  __device__ __forceinline__ void load_cg(const float* p) {
    if constexpr (VW == 4) {
      const float4 t = __ldcg(reinterpret_cast<const float4*>(p));
      v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else if constexpr (VW == 2) {
      const float2 t = __ldcg(reinterpret_cast<const float2*>(p));
      v[0] = t.x; v[1] = t.y;
    } else {
      v[0] = __ldcg(p);
    }
  }
  __device__ __forceinline__ void load(const float* p) {   // shared memory
    if constexpr (VW == 4) {
      const float4 t = *reinterpret_cast<const float4*>(p);
      v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else if constexpr (VW == 2) {
      const float2 t = *reinterpret_cast<const float2*>(p);
      v[0] = t.x; v[1] = t.y;
    } else {
      v[0] = *p;
    }
  }
  __device__ __forceinline__ void store(float* p) const {
    if constexpr (VW == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    else if constexpr (VW == 2) *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
    else *p = v[0];
  }
};

struct Args {
  const float* rec;   // matrix-free point records (MF_REC floats per GLL point)
  const int* ge;      // dof map of the operator elements
  int nelmt;
  const int* pos;     // gather position of each element slot
  const int* gptr;    // gather groups: slot range and dof numbers
  const int* gdof;
  int ngroups;
  float *u, *r, *z, *p, *kp, *Y;
  const float* dp;    // inverted diagonal
  ColState* cs;
  PcgGlobal* G;       // cntB counts the barrier's arrivals
  float4* part;       // block partials (three floats): phase B [KR][grid], phase C [2 KR][grid]
  const float* f;     // right-hand side of a new solve
  PersistStart st;
  PersistOut* out;    // pinned host memory
  int chunk;          // iterations to run
  int cached;         // elements whose maps and records a block keeps in shared memory
};

template <int KR>
struct Shape {
  static constexpr int VW = KR < 4 ? KR : 4;     // columns per piece
  static constexpr int QPD = KR / VW;            // pieces per dof row
  static constexpr int LPN = 3 * QPD;            // pieces per node
  static constexpr int UF = NEDOF * VW;          // shared floats per warp: p of the element
  static constexpr int FF = NGLL * 9 * VW;       //   and the fluxes at its points
  static constexpr size_t SMEM = (size_t)NWARP * (UF + FF) * sizeof(float);
  static constexpr int EF = NGLL * (MF_REC + 4);  // words per cached element: records, maps {dof x 3, position}
  static constexpr int CACHE = (int)((220 * 1024 - SMEM) / (EF * sizeof(float)));
  static_assert(NT % LPN == 0, "a thread keeps its columns");
};

__device__ __forceinline__ float dcoef(int i, int t) {   // D[i][t] of the GLL points -1, 0, 1
  return i == 0 ? (t == 0 ? -1.5f : t == 1 ? 2.0f : -0.5f)
                : i == 1 ? (t == 0 ? -0.5f : t == 1 ? 0.0f : 0.5f) : (t == 0 ? 0.5f : t == 1 ? -2.0f : 1.5f);
}

// Element products of one warp: element e, columns c0 .. c0 + VW - 1.
template <int KR>
__device__ __forceinline__ void element_product(const Args& A, int e, const float* cache, int c0, int lane,
                                                const float (&beta)[Shape<KR>::VW], float* U, float* F) {
  using S = Shape<KR>;
  constexpr int VW = S::VW;
  const int a = lane;
  Vec<VW> u[3];
  int q = -1;
  float Ji[9], c11 = 0.f, c12 = 0.f, c44 = 0.f;
  if (a < NGLL) {
    int gd[3];
    float4 r0, r1, r2;
    if (cache) {
      const float4* Rp = reinterpret_cast<const float4*>(cache) + 4 * a;
      const int4 m = *reinterpret_cast<const int4*>(Rp + 3);
      r0 = Rp[0]; r1 = Rp[1]; r2 = Rp[2];
      gd[0] = m.x; gd[1] = m.y; gd[2] = m.z; q = m.w;
    } else {
#pragma unroll
      for (int c = 0; c < 3; ++c) gd[c] = __ldg(A.ge + (size_t)e * NEDOF + 3 * a + c);
      q = __ldg(A.pos + (size_t)e * NGLL + a);
      const float4* Rp = reinterpret_cast<const float4*>(A.rec + ((size_t)e * NGLL + a) * MF_REC);
      r0 = __ldg(Rp); r1 = __ldg(Rp + 1); r2 = __ldg(Rp + 2);
    }
    Ji[0] = r0.x; Ji[1] = r0.y; Ji[2] = r0.z; Ji[3] = r0.w; Ji[4] = r1.x; Ji[5] = r1.y; Ji[6] = r1.z; Ji[7] = r1.w;
    Ji[8] = r2.x; c11 = r2.y; c12 = r2.z; c44 = r2.w;
    Vec<VW> pv[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      pv[c].load_cg(A.p + (size_t)gd[c] * KR + c0);
      u[c].load_cg(A.z + (size_t)gd[c] * KR + c0);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
#pragma unroll
      for (int k = 0; k < VW; ++k) u[c].v[k] = fmaf(beta[k], pv[c].v[k], u[c].v[k]);
      u[c].store(U + (3 * a + c) * VW);
    }
  }
  __syncwarp();
  const int ic[3] = {a % 3, (a / 3) % 3, a / 9};
  if (a < NGLL) {
    // reference gradient gr[c][r], the line's nodes in order
    Vec<VW> gr[3][3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      constexpr int st[3] = {1, 3, 9};
      const float* ul = U + 3 * (a - ic[r] * st[r]) * VW;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
#pragma unroll
        for (int tt = 0; tt < 3; ++tt) {
          const float d = dcoef(ic[r], tt);
          Vec<VW> x;
          x.load(ul + (3 * tt * st[r] + c) * VW);
#pragma unroll
          for (int k = 0; k < VW; ++k) gr[c][r].v[k] = tt == 0 ? d * x.v[k] : fmaf(d, x.v[k], gr[c][r].v[k]);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < VW; ++k) {
      float gp[3][3], T[3][3];
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int d = 0; d < 3; ++d)
          gp[c][d] = fmaf(Ji[3 * d], gr[c][0].v[k], fmaf(Ji[3 * d + 1], gr[c][1].v[k], Ji[3 * d + 2] * gr[c][2].v[k]));
      T[0][0] = fmaf(c11, gp[0][0], c12 * (gp[1][1] + gp[2][2]));
      T[1][1] = fmaf(c11, gp[1][1], c12 * (gp[0][0] + gp[2][2]));
      T[2][2] = fmaf(c11, gp[2][2], c12 * (gp[0][0] + gp[1][1]));
      T[0][1] = T[1][0] = c44 * (gp[0][1] + gp[1][0]);
      T[1][2] = T[2][1] = c44 * (gp[1][2] + gp[2][1]);
      T[0][2] = T[2][0] = c44 * (gp[0][2] + gp[2][0]);
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int r = 0; r < 3; ++r)
          gr[c][r].v[k] = fmaf(Ji[r], T[c][0], fmaf(Ji[3 + r], T[c][1], Ji[6 + r] * T[c][2]));
    }
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int r = 0; r < 3; ++r) gr[c][r].store(F + (9 * a + 3 * r + c) * VW);
  }
  __syncwarp();
  if (a < NGLL) {
    // rows of node a: the xi, eta and zeta fluxes of its lines in order
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      constexpr int st[3] = {1, 3, 9};
      const float* fl = F + (9 * (a - ic[r] * st[r]) + 3 * r) * VW;
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int tt = 0; tt < 3; ++tt) {
          const float d = dcoef(tt, ic[r]);
          Vec<VW> x;
          x.load(fl + (9 * tt * st[r] + c) * VW);
#pragma unroll
          for (int k = 0; k < VW; ++k) u[c].v[k] = r == 0 && tt == 0 ? d * x.v[k] : fmaf(d, x.v[k], u[c].v[k]);
        }
    }
    if (q >= 0) {
      float* dst = A.Y + (size_t)q * 3 * KR + c0;
#pragma unroll
      for (int c = 0; c < 3; ++c) u[c].store(dst + c * KR);
    }
  }
}

// R pieces per thread in registers; STREAMED_FEW: up to four, STREAMED: any number, streamed.
constexpr int STREAMED_FEW = 0, STREAMED = -1;
template <int KR, int R>
__global__ void __launch_bounds__(NT, 1) k_pcg_persistent(Args A) {
  using S = Shape<KR>;
  constexpr int VW = S::VW, QPD = S::QPD, LPN = S::LPN;
  constexpr int RR = R > 0 ? R : 1;
  // A thread's products of a column: up to four in two floats; three keep the
  // rounding errors of many.  (3,289 elements, 8 columns: 27.8 us an iteration, 28.7
  // with three floats there too.)
  using Dot = std::conditional_t<R != STREAMED && R <= 4, CompSum, CompSum3>;
  extern __shared__ __align__(16) float smem[];
  __shared__ Sum3 sred[2 * KR][NWARP];
  // block-local copy of the column state (identical in every block)
  __shared__ Sum3 c_rz[KR], c_rr[KR], c_goal[KR];
  __shared__ Sum3 c_pkp[KR];
  __shared__ float c_alpha[KR], c_beta[KR];
  __shared__ int c_live[KR], c_ran[KR], c_iters[KR], c_failed[KR];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  PcgGlobal* G = A.G;
  const int init = A.st.init, keep = A.st.keep, maxiter = A.st.maxiter, kcols = A.st.kcols;
  if (!init && G->all_done) return;
  if (t < KR) {
    const ColState c = A.cs[t];
    c_rz[t] = split3(c.rz);
    c_live[t] = (A.st.active >> t) & 1u;
    if (!init) {
      c_alpha[t] = (float)c.alpha; c_beta[t] = (float)c.beta; c_rr[t] = split3(c.rr);
      c_goal[t] = split3(c.tol * c.tol * c.rr0);   // |r|^2 at which the column stops
      c_live[t] = c_live[t] && !c.done; c_iters[t] = c.iters; c_failed[t] = c.failed;
    } else {
      c_alpha[t] = c_beta[t] = 0.f;
      c_rr[t] = c_goal[t] = zero3();
      c_iters[t] = c_failed[t] = 0;
    }
    c_ran[t] = c_live[t];
  }
  int itn = init ? 0 : G->it, alldone = 0;
  const int grid = gridDim.x, bid = blockIdx.x;
  unsigned arrivals = 0;

  // nodes of a block and pass; with no more pieces than threads every block has its
  // share, and the warps without a piece leave the sums to the others
  const int npb = R == 1 ? (A.ngroups + grid - 1) / grid : NT / LPN;
  const int nwarp = R == 1 ? (npb * LPN + 31) / 32 : NWARP;

  // Grid barrier: earlier writes of the block are visible to every block
  // after it.  Returns false when the wait ran out.
  auto barrier = [&]() -> bool {
    __syncthreads();
    bool good = true;
    if (t == 0) {
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&G->cntB) : "memory");
      arrivals += (unsigned)grid;
      unsigned n;
      int tries = 0;
      do {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(n) : "l"(&G->cntB) : "memory");
        if (++tries > POLL_TRIES) good = false;
      } while (n < arrivals && good);
      if (!good) atomicExch(&G->err, 1);
    }
    return !__syncthreads_or(!good);
  };
  // sred[v][warp] summed over warps into this block's column of the partials
  // (the maximum of the high parts when MAXOP)
  auto publish = [&](auto nvc, auto maxc, float4* out) {
    constexpr int NV = decltype(nvc)::value;
    constexpr bool MAXOP = decltype(maxc)::value;
    __syncthreads();
    constexpr int SUB = 8, NVW = 32 / SUB;   // lanes a value, values a warp
    static_assert((NV + NVW - 1) / NVW <= NWARP && SUB <= NWARP, "warps and their lanes");
    if (warp < (NV + NVW - 1) / NVW) {
      const int v = warp * NVW + lane / SUB, s = lane % SUB;
      Sum3 x[1] = {zero3()};
      if (v < NV) {
        if (s < nwarp) x[0] = sred[v][s];
        for (int w = s + SUB; w < nwarp; w += SUB) {
          if (MAXOP) x[0].h = fmaxf(x[0].h, sred[v][w].h);
          else x[0].add(sred[v][w]);
        }
      }
      if (MAXOP) {
#pragma unroll
        for (int o = SUB / 2; o >= 1; o >>= 1) x[0].h = fmaxf(x[0].h, __shfl_xor_sync(0xffffffffu, x[0].h, o));
      } else {
        Reduce<1, SUB / 2, 1>::run(x, lane);
      }
      if (v < NV && s == 0) __stcg(out + (size_t)v * grid + bid, make_float4(x[0].h, x[0].l, x[0].m, 0.f));
    }
  };
  // sum over the blocks of one value's partials, by one warp
  auto block_sum = [&](const float4* in) -> Sum3 {
    constexpr int NB = (MAX_BLOCKS + 31) / 32;
    Sum3 w[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      const float4 v = lane + 32 * i < grid ? __ldcg(in + lane + 32 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
      w[i] = Sum3{v.x, v.y, v.z};
    }
#pragma unroll
    for (int o = 1; o < NB; o *= 2)
#pragma unroll
      for (int i = 0; i + o < NB; i += 2 * o) w[i].add(w[i + o]);
    Sum3 x[1] = {w[0]};
    Reduce<1, 16, 1>::run(x, lane);
    return norm3(x[0]);
  };

  // product m of a thread
  auto dot_add = [](auto& x, int m, float a, float b) {
    if constexpr (R > 0 && std::is_same_v<Dot, CompSum>) {
      if (m == 0) { x.set(a, b); return; }
    }
    x.add(a, b);
  };

  // the thread's pieces: columns c0 .. c0 + VW - 1 of dof row d of nodes g0, g0 + gstride, ...
  const int qp = t % LPN, d = qp / QPD, c0 = VW * (qp % QPD);
  const int gstride = grid * (NT / LPN);
  // consecutive nodes stay in one block
  const int g0 = t / LPN < npb ? bid * npb + t / LPN : A.ngroups;
  Vec<VW> ru[RR], rr[RR], rp[RR], rk[RR];
  int gd[RR], sa[RR], sb[RR];
  float dv[RR];
  if constexpr (R > 0) {
#pragma unroll
    for (int m = 0; m < R; ++m) {
      const int g = g0 + m * gstride;
      gd[m] = g < A.ngroups ? A.gdof[3 * g + d] : 0;
      sa[m] = g < A.ngroups ? A.gptr[g] : 0;
      sb[m] = g < A.ngroups ? A.gptr[g + 1] : 0;
      dv[m] = A.dp[gd[m]];
      const size_t o = (size_t)gd[m] * KR + c0;
      rp[m].zero();
      if (init) {
        ru[m].zero();
        rr[m].load_cg(A.f + o);
        if (keep) rp[m].load_cg(A.p + o);
      } else {
        ru[m].load_cg(A.u + o);
        rr[m].load_cg(A.r + o);
        rp[m].load_cg(A.p + o);
      }
    }
  }
  float* U = smem + (size_t)warp * (S::UF + S::FF);
  float* F = U + S::UF;
  float4* partB = A.part;
  float4* partC = A.part + (size_t)grid * KR;
  // the block's run of (element, column group) pairs
  const int nw = A.nelmt * QPD, per = (nw + grid - 1) / grid, w0 = bid * per, w1 = min(nw, w0 + per);
  float* cache = smem + (size_t)NWARP * (S::UF + S::FF);
  const int e0 = w0 / QPD;
  for (int i = t; i < A.cached * NGLL; i += NT) {
    const int e = e0 + i / NGLL, a = i % NGLL;
    if (e >= A.nelmt) break;
    float4* o = reinterpret_cast<float4*>(cache) + 4 * i;
    const float4* Rp = reinterpret_cast<const float4*>(A.rec + ((size_t)e * NGLL + a) * MF_REC);
    const int* g = A.ge + (size_t)e * NEDOF + 3 * a;
    o[0] = Rp[0]; o[1] = Rp[1]; o[2] = Rp[2];
    *reinterpret_cast<int4*>(o + 3) = make_int4(g[0], g[1], g[2], A.pos[(size_t)e * NGLL + a]);
  }
  __syncthreads();

  // warp sums of the thread's values (x[i] of column VW r + i % VW, r = lane
  // class) into sred[(i / VW) KR + column][warp]
  auto reduce_lanes = [&](auto& dots) {
    constexpr int N = sizeof(dots) / sizeof(dots[0]);
    if (warp >= nwarp) return;
    Sum3 x[N];
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = dots[i].sum();
    constexpr int LOGN = N == 8 ? 3 : N == 4 ? 2 : N == 2 ? 1 : 0;
    Reduce<N, 16, QPD>::run(x, lane);
    // bit 4 of the lane chose the upper half of the values, bit 3 of that half, ...
    const int i = N == 1 ? 0 : lane >> (5 - LOGN), rest = lane & ((32 >> LOGN) - 1);
    if (rest < QPD) sred[(i / VW) * KR + VW * rest + i % VW][warp] = x[0];
  };
  // kp of one piece: the node's slots in element order, four loads in flight
  auto slot_sum = [&](int a, int b, Vec<VW>& acc) {
    const float* y = A.Y + VW * qp;
    acc.zero();
    for (int s0 = a; s0 < b; s0 += 4) {
      Vec<VW> v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (s0 + k < b) v[k].load_cg(y + (size_t)(s0 + k) * 3 * KR);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (s0 + k < b)
#pragma unroll
          for (int c = 0; c < VW; ++c) acc.v[c] = acc.v[c] + v[k].v[c];
    }
  };

  // r.z and r.r of the thread's columns over the grid, then each column's step,
  // identical in every block: the start of a solve, or stop test and beta
  auto column_steps = [&](Dot (&zz)[2 * VW], bool first) -> bool {
    reduce_lanes(zz);
    publish(std::integral_constant<int, 2 * KR>{}, std::false_type{}, partC);
    if (!barrier()) return false;
    for (int j = warp; j < KR; j += NWARP) {
      const Sum3 x = block_sum(partC + (size_t)j * grid), y = block_sum(partC + (size_t)(KR + j) * grid);
      if (lane == 0 && c_live[j]) {
        c_rr[j] = y;
        if (first) {
          if (keep) c_beta[j] = div3(x, c_rz[j]);
          c_rz[j] = x;
          c_goal[j] = split3(A.st.tol * A.st.tol * y.value());
        } else if (at_most(y, c_goal[j])) {
          c_live[j] = 0; c_iters[j] = itn;
        } else if (itn >= maxiter) {
          c_live[j] = 0; c_failed[j] = 1; c_iters[j] = maxiter + 1;
        } else {
          c_beta[j] = div3(x, c_rz[j]);
          c_rz[j] = x;
        }
      }
    }
    __syncthreads();
    return true;
  };

  // ---- a new solve: u = 0, r = f, z = D r, and p = 0 unless the last solve's
  // direction is continued (beta = r.z / the last r.z) ----
  if (init) {
    Dot zz[2 * VW];
    if (bid == 0 && t < KR) { A.u[t] = 0.f; A.r[t] = 0.f; A.z[t] = 0.f; A.p[t] = 0.f; }   // constrained dofs
    auto start = [&](size_t o, float D, const Vec<VW>& rv, int m) {
      Vec<VW> zv;
#pragma unroll
      for (int q = 0; q < VW; ++q) {
        zv.v[q] = D * rv.v[q];
        dot_add(zz[q], m, rv.v[q], zv.v[q]);
        dot_add(zz[VW + q], m, rv.v[q], rv.v[q]);
      }
      zv.store(A.z + o);
      if (!keep) {
        Vec<VW> none;
        none.zero();
        none.store(A.p + o);
      }
    };
    if constexpr (R > 0) {
#pragma unroll
      for (int m = 0; m < R; ++m)
        if (gd[m]) start((size_t)gd[m] * KR + c0, dv[m], rr[m], m);
    } else {
      for (int g = g0; g < A.ngroups; g += gstride) {
        const int gq = __ldg(A.gdof + 3 * g + d);
        if (!gq) continue;
        const size_t o = (size_t)gq * KR + c0;
        Vec<VW> rv, none;
        none.zero();
        rv.load_cg(A.f + o);
        none.store(A.u + o);
        rv.store(A.r + o);
        start(o, __ldg(A.dp + gq), rv, 1);
      }
    }
    if (!column_steps(zz, true)) return;
  }

  for (int k = 0; k < A.chunk; ++k) {
    // ---- A: element products ----
    for (int w = w0 + warp; w < w1; w += NWARP) {
      const int e = w / QPD, cc = VW * (w - e * QPD);
      float beta[VW];
#pragma unroll
      for (int q = 0; q < VW; ++q) beta[q] = c_beta[cc + q];
      element_product<KR>(A, e, e - e0 < A.cached ? cache + (size_t)(e - e0) * S::EF : nullptr, cc, lane, beta, U, F);
      __syncwarp();
    }
    if (!barrier()) return;
    // ---- B: kp, p and p.kp ----
    bool live[VW];
    float beta[VW];
    Dot dot[VW];
#pragma unroll
    for (int q = 0; q < VW; ++q) { live[q] = c_live[c0 + q] != 0; beta[q] = c_beta[c0 + q]; }
    if constexpr (R > 0) {
#pragma unroll
      for (int m = 0; m < R; ++m) {
        slot_sum(sa[m], sb[m], rk[m]);
        if (!gd[m]) continue;
#pragma unroll
        for (int q = 0; q < VW; ++q)
          if (live[q]) {
            // z = D r as phase C formed it
            rp[m].v[q] = fmaf(beta[q], rp[m].v[q], dv[m] * rr[m].v[q]);
            dot_add(dot[q], m, rp[m].v[q], rk[m].v[q]);
          }
        rp[m].store(A.p + (size_t)gd[m] * KR + c0);
      }
    } else {
      for (int g = g0; g < A.ngroups; g += gstride) {
        const int gq = __ldg(A.gdof + 3 * g + d);
        const size_t o = (size_t)gq * KR + c0;
        Vec<VW> pv, zv, acc;
        pv.load_cg(A.p + o);
        zv.load_cg(A.z + o);
        slot_sum(__ldg(A.gptr + g), __ldg(A.gptr + g + 1), acc);
        if (!gq) continue;
#pragma unroll
        for (int q = 0; q < VW; ++q)
          if (live[q]) {
            pv.v[q] = fmaf(beta[q], pv.v[q], zv.v[q]);
            dot[q].add(pv.v[q], acc.v[q]);
          }
        pv.store(A.p + o);
        acc.store(A.kp + o);
      }
    }
    reduce_lanes(dot);
    publish(std::integral_constant<int, KR>{}, std::false_type{}, partB);
    if (!barrier()) return;
    for (int j = warp; j < KR; j += NWARP) {
      const Sum3 x = block_sum(partB + (size_t)j * grid);
      if (lane == 0 && c_live[j]) { c_alpha[j] = div3(c_rz[j], x); c_pkp[j] = x; }
    }
    __syncthreads();
    // ---- C: u, r, z and r.z, r.r ----
    float alpha[VW];
    Dot zz[2 * VW];   // r.z of the thread's columns, then r.r
#pragma unroll
    for (int q = 0; q < VW; ++q) alpha[q] = live[q] ? c_alpha[c0 + q] : 0.f;
    if constexpr (R > 0) {
#pragma unroll
      for (int m = 0; m < R; ++m) {
        if (!gd[m]) continue;
        Vec<VW> zv;
#pragma unroll
        for (int q = 0; q < VW; ++q) {
          if (live[q]) {
            ru[m].v[q] = fmaf(alpha[q], rp[m].v[q], ru[m].v[q]);
            rr[m].v[q] = fmaf(-alpha[q], rk[m].v[q], rr[m].v[q]);
          }
          zv.v[q] = dv[m] * rr[m].v[q];
          dot_add(zz[q], m, rr[m].v[q], zv.v[q]);
          dot_add(zz[VW + q], m, rr[m].v[q], rr[m].v[q]);
        }
        zv.store(A.z + (size_t)gd[m] * KR + c0);
      }
    } else {
      for (int g = g0; g < A.ngroups; g += gstride) {
        const int gq = __ldg(A.gdof + 3 * g + d);
        if (!gq) continue;
        const size_t o = (size_t)gq * KR + c0;
        const float D = __ldg(A.dp + gq);
        Vec<VW> pv, uv, rv, kv, zv;
        pv.load_cg(A.p + o);
        uv.load_cg(A.u + o);
        rv.load_cg(A.r + o);
        kv.load_cg(A.kp + o);
#pragma unroll
        for (int q = 0; q < VW; ++q) {
          if (live[q]) {
            uv.v[q] = fmaf(alpha[q], pv.v[q], uv.v[q]);
            rv.v[q] = fmaf(-alpha[q], kv.v[q], rv.v[q]);
          }
          zv.v[q] = D * rv.v[q];
          zz[q].add(rv.v[q], zv.v[q]);
          zz[VW + q].add(rv.v[q], rv.v[q]);
        }
        uv.store(A.u + o);
        rv.store(A.r + o);
        zv.store(A.z + o);
      }
    }
    ++itn;
    if (!column_steps(zz, false)) return;
    alldone = !__syncthreads_or(t < kcols && c_live[t < KR ? t : 0]);
    if (alldone) break;
  }

  // max|p| of each column's last step (a stopped column keeps its direction)
  float mp[VW];
#pragma unroll
  for (int q = 0; q < VW; ++q) mp[q] = 0.f;
  if constexpr (R > 0) {
#pragma unroll
    for (int m = 0; m < R; ++m) {
      if (!gd[m]) continue;
      const size_t o = (size_t)gd[m] * KR + c0;
      ru[m].store(A.u + o);
      rr[m].store(A.r + o);
#pragma unroll
      for (int q = 0; q < VW; ++q) mp[q] = fmaxf(mp[q], fabsf(rp[m].v[q]));
    }
  } else {
    for (int g = g0; g < A.ngroups; g += gstride) {
      const int gq = __ldg(A.gdof + 3 * g + d);
      if (!gq) continue;
      Vec<VW> pv;
      pv.load_cg(A.p + (size_t)gq * KR + c0);
#pragma unroll
      for (int q = 0; q < VW; ++q) mp[q] = fmaxf(mp[q], fabsf(pv.v[q]));
    }
  }
#pragma unroll
  for (int q = 0; q < VW; ++q) {
#pragma unroll
    for (int o = 16; o >= QPD; o >>= 1) mp[q] = fmaxf(mp[q], __shfl_xor_sync(0xffffffffu, mp[q], o));
    if (lane < QPD) sred[VW * lane + q][warp].h = mp[q];
  }
  publish(std::integral_constant<int, KR>{}, std::true_type{}, partB);
  if (!barrier()) return;
  // the column state leaves with block 0
  if (bid == 0) {
    if (t < KR) {
      ColState& c = A.cs[t];
      float m = 0.f;
      for (int b = 0; b < grid; ++b) m = fmaxf(m, __ldcg(partB + (size_t)t * grid + b).x);
      c.active = (A.st.active >> t) & 1u;
      if (c.active) {
        // a column that has stopped keeps the r.z that its last step took
        if (c_live[t]) c.alpha = c_alpha[t];
        else if (c_ran[t]) c.alpha = c_rz[t].value() / c_pkp[t].value();
        c.rz = c_rz[t].value(); c.beta = c_beta[t]; c.rr = c_rr[t].value();
        c.maxp = m; c.done = !c_live[t]; c.iters = c_iters[t]; c.failed = c_failed[t];
        if (init) { c.tol = 1.0; c.rr0 = c_goal[t].value(); }   // their product is the goal
        A.out->iters[t] = c_iters[t];
        A.out->step[t] = fabs(c.alpha) * (double)m;
      }
    }
    if (t == 0) {
      G->it = itn;
      G->all_done = alldone;
      A.out->it = itn;
      A.out->state = alldone ? PERSIST_DONE : PERSIST_MORE;
    }
  }
}

}  // namespace pp

// Largest mesh that takes the persistent chunk: where a phase has more work
// than 15 warps per SM hide, separate launches with their own register budgets
// win.  us per iteration of a whole trial, persistent against separate kernels:
//   elements   1 column       2 columns      4 columns      8 columns      16 columns
//    1,071    9.5 /  28.0   10.9 /  29.9   13.0 /  33.5   17.5 /  35.9    29.8 /  41.8
//    2,662                                                                53.8 /  58.1
//    3,289   12.3 /  34.5   14.9 /  38.6   20.2 /  37.9   34.5 /  45.4    61.5 /  61.1
//    5,488   14.9 /  40.5   18.2 /  43.2   26.4 /  45.4   47.8 /  55.0    84.2 /  75.5 (5,040)
//    7,056                                                58.2 /  58.1
//    9,600   19.7 /  47.2   25.3 /  49.3   40.6 /  49.5   72.9 /  65.8
//   12,000   22.8 /  50.0   32.7 /  53.9   50.0 /  56.8
//   18,000                                 68.3 /  67.1
//   25,000   43.3 /  67.1   57.6 /  79.0
//   43,200                 111.2 / 111.1
//   53,760  100.7 / 105.9
//   58,032  113.7 / 111.9
int persist_max_elements(int KR) {
  return KR == 1 ? 57000 : KR == 2 ? 42500 : KR == 4 ? 17000 : KR == 8 ? 7000 : 3000;
}

bool persist_enabled() {
  static const bool on = !(getenv("SG_PERSIST") && atoi(getenv("SG_PERSIST")) == 0);
  return on;
}

int persist_iterations(int n) {
  static const int set = getenv("SG_PERSIST_CHUNK") ? atoi(getenv("SG_PERSIST_CHUNK")) : 0;
  return set > 0 ? set : n;
}

template <int KR, int R>
static bool launch_persistent(const pp::Args& A, int grid, size_t smem, cudaStream_t s) {
  static std::atomic<unsigned long long> allowed{};
  if (!allow_smem(allowed, (const void*)pp::k_pcg_persistent<KR, R>, 220 * 1024)) {
    cudaGetLastError();
    return false;
  }
  pp::Args a = A;
  void* args[] = {&a};
  if (cudaLaunchCooperativeKernel((const void*)pp::k_pcg_persistent<KR, R>, grid, pp::NT, args, smem, s) !=
      cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  add_launches(1);
  return true;
}

// Up to `chunk` PCG iterations of the FP32 solve (residual test) as one
// cooperative launch; st says whether a new solve begins.  Returns false when
// the launch is not possible (the caller then runs the separate kernels).
template <int KR>
bool launch_pcg_persistent(const float* rec, const int* ge, int nelmt, const int* pos, const GatherTopo& T,
                           const float* f, float* u, float* r, float* z, float* p, float* kp, float* Y,
                           const float* dp, ColState* cs, PcgGlobal* G, double* part, const PersistStart& st,
                           PersistOut* out, int chunk, cudaStream_t s) {
  using S = pp::Shape<KR>;
  // one block per SM, fewer where that still gives every scheduler of the
  // SMs in use no more than one warp of phase A
  long warps = (long)nelmt * S::QPD, pieces = (long)T.ngroups * S::LPN;
  long grid = (warps + 3) / 4;
  if (grid < (pieces + pp::NT - 1) / pp::NT) grid = (pieces + pp::NT - 1) / pp::NT;
  if (grid > pp::MAX_BLOCKS) grid = pp::MAX_BLOCKS;
  if (grid < 1) return false;
  const long per = (pieces + grid * pp::NT - 1) / (grid * pp::NT);   // pieces per thread
  static_assert((size_t)pp::MAX_BLOCKS * 3 * KR * sizeof(float4) <= (size_t)NPART * 16 * 2 * sizeof(double),
                "partials fit half the buffer");
  if (st.init) cudaMemsetAsync(G, 0, sizeof(PcgGlobal), s);
  else cudaMemsetAsync(&G->cntB, 0, sizeof(unsigned), s);
  // elements a block works on: its run of pairs touches at most this many
  const long runs = (warps + grid - 1) / grid;
  long cached = (runs + S::QPD - 1) / S::QPD + (S::QPD > 1 ? 1 : 0);
  if (cached > S::CACHE) cached = S::CACHE;
  const size_t smem = S::SMEM + (size_t)cached * S::EF * sizeof(float);
  const pp::Args A{rec, ge, nelmt, pos, T.d_ptr, T.d_dof, T.ngroups, u, r, z, p, kp, Y, dp, cs, G,
                   reinterpret_cast<float4*>(part), f, st, out, chunk, (int)cached};
  if (per <= 1) return launch_persistent<KR, 1>(A, (int)grid, smem, s);
  if (per <= 2) return launch_persistent<KR, 2>(A, (int)grid, smem, s);
  if constexpr (KR <= 2)
    if (per <= 4) return launch_persistent<KR, 4>(A, (int)grid, smem, s);
  if constexpr (KR == 1)
    if (per <= 8) return launch_persistent<KR, 8>(A, (int)grid, smem, s);
  if constexpr (KR > 2)
    if (per <= 4) return launch_persistent<KR, pp::STREAMED_FEW>(A, (int)grid, smem, s);
  return launch_persistent<KR, pp::STREAMED>(A, (int)grid, smem, s);
}

#define SG_PP_INST(KR)                                                                                             \
  template bool launch_pcg_persistent<KR>(const float*, const int*, int, const int*, const GatherTopo&,            \
                                          const float*, float*, float*, float*, float*, float*, float*,            \
                                          const float*, ColState*, PcgGlobal*, double*, const PersistStart&,       \
                                          PersistOut*, int, cudaStream_t);
SG_PP_INST(1)
SG_PP_INST(2)
SG_PP_INST(4)
SG_PP_INST(8)
SG_PP_INST(16)

}  // namespace sg
