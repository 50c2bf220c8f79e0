// Grouped FP64 / complex128 GEMM over all tasks of one contraction.
//
// Replaces the reference's serial loop of one cblas_dgemm / cublasDgemm per task with
// beta = 0 for the first task of an output block and beta = 1 after it
// (global_operations.h:895-992 -> raw_data_operations.h:530-548 -> blas_level3.h:35-56,
// :797-856). Every output tile is owned by one warp that loops over all tasks of its output
// block, accumulating sign_t * A_t[tile rows, :] B_t[:, tile cols] in registers, and stores
// the tile once: no read-modify-write of C, no atomics, deterministic.
//
// Two kernels, chosen per output block when the plan is built:
//  * k_gemm_f64    - FP64 / complex128 (4 real FMAs per complex FMA) on warp tiles. On this
//                    GPU the FP64 tensor path (mma.sync m8n8k4 f64) runs at the same rate as
//                    DFMA (about 1.05 TFLOP/s each, measured) but pads every block to 8 x 8 x 4
//                    fragments, so DFMA, with nothing predicated, is the faster FP64 kernel;
//  * k_gemm_skinny - output blocks with n <= 8 and k <= 8 (the MPO steps of the two-site
//                    matvec: m up to 3e4, k, n <= 3): one output per lane, memory-streaming.
#include <algorithm>

#include "ctrct.h"

namespace qltg {
namespace {

constexpr int NT = 128;            // threads of an FP64 GEMM CTA: one warp per sub-partition
// 16 warps per SM hide the operand latency (2 / 3 / 4 CTAs at D = 4000: 3.02 / 2.60 / 2.52 ms)
constexpr int kF64CtasPerSm = 4;

__device__ __forceinline__ void fma_acc(double& acc, double a, double b) { acc = fma(a, b, acc); }
__device__ __forceinline__ void fma_acc(double2& acc, double2 a, double2 b) {
  acc.x = fma(a.x, b.x, acc.x);
  acc.x = fma(-a.y, b.y, acc.x);
  acc.y = fma(a.x, b.y, acc.y);
  acc.y = fma(a.y, b.x, acc.y);
}
__device__ __forceinline__ double zero_of(double) { return 0.0; }
__device__ __forceinline__ double2 zero_of(double2) { return make_double2(0.0, 0.0); }
// Multiply by a +-1 sign without touching the FP64 pipe: flip the IEEE sign bit(s).
__device__ __forceinline__ double flip(double x, unsigned long long m) {
  return __longlong_as_double(__double_as_longlong(x) ^ (long long)m);
}
__device__ __forceinline__ double2 flip(double2 x, unsigned long long m) { return make_double2(flip(x.x, m), flip(x.y, m)); }
__device__ __forceinline__ unsigned long long sign_mask(int sign) { return sign < 0 ? 0x8000000000000000ull : 0ull; }

// One task added to a warp's 8 TM x 4 TN tile: lane (lr, lc) of the warp's 8 x 4 grid holds the
// outputs (lr + 8 i, lc + 4 j). Operands go straight from L1 / L2 into registers, U values of k
// ahead of their use (the next values of an A row share its cache line; four B columns are one
// sector). A predicated-off FP64 instruction takes as long as an executed one (78 cycles on its
// sub-partition, measured), so nothing here is predicated: tiles are instantiated per number of
// pieces inside the block, and a task's last k % U values run in a loop of their own.
template <typename T, int TM, int TN>
__device__ __forceinline__ void f64_tile_task(T (&acc)[TM][TN], const T* __restrict__ a, const T* __restrict__ b, int k,
                                              int n, unsigned long long sg, const int (&row)[TM],
                                              const int (&col)[TN]) {
  constexpr int U = (sizeof(T) == 8 ? 4 : 2) * (TN == 1 ? 2 : 1) / TM;
  T av[U][TM], bv[U][TN];
  auto load = [&](int k0) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int i = 0; i < TM; ++i) av[u][i] = __ldg(a + (int64_t)row[i] * k + k0 + u);
#pragma unroll
      for (int j = 0; j < TN; ++j) bv[u][j] = __ldg(b + (int64_t)(k0 + u) * n + col[j]);
    }
  };
  int k0 = 0;
  if (U <= k) load(0);
  for (; k0 + U <= k; k0 += U) {
    T ac[U][TM], bc[U][TN];
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int i = 0; i < TM; ++i) ac[u][i] = flip(av[u][i], sg);
#pragma unroll
      for (int j = 0; j < TN; ++j) bc[u][j] = bv[u][j];
    }
    if (k0 + 2 * U <= k) load(k0 + U);
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) fma_acc(acc[i][j], ac[u][i], bc[u][j]);
  }
#pragma unroll 1
  for (; k0 < k; ++k0) {
    T ac[TM], bc[TN];
#pragma unroll
    for (int i = 0; i < TM; ++i) ac[i] = flip(__ldg(a + (int64_t)row[i] * k + k0), sg);
#pragma unroll
    for (int j = 0; j < TN; ++j) bc[j] = __ldg(b + (int64_t)k0 * n + col[j]);
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) fma_acc(acc[i][j], ac[i], bc[j]);
  }
}

// All tasks of an output block added up for the tile of 8 TM rows and 4 TN columns at (r0, c0),
// every 8 x 4 piece of which holds outputs of the block, by one warp, and stored. A function of
// its own: inlined side by side the sizes' prefetch registers spill.
template <typename T, int TM, int TN>
__device__ __noinline__ void f64_tile(const GemmCBlk& cb, const GemmTask* __restrict__ task, int r0, int c0, int lane,
                                         const T* __restrict__ A, const T* __restrict__ As, const T* __restrict__ B,
                                         const T* __restrict__ Bs, T* __restrict__ C) {
  const int lr = lane >> 2, lc = lane & 3, m = cb.m, n = cb.n;
  int row[TM], col[TN];  // this lane's rows and columns, clamped into the block
#pragma unroll
  for (int i = 0; i < TM; ++i) row[i] = min(r0 + 8 * i + lr, m - 1);
#pragma unroll
  for (int j = 0; j < TN; ++j) col[j] = min(c0 + 4 * j + lc, n - 1);
  T acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = zero_of(T());
  for (int t = cb.t0; t < cb.t1; ++t) {
    const GemmTask tk = task[t];
    f64_tile_task<T, TM, TN>(acc, operand_block(A, As, tk.a_off), operand_block(B, Bs, tk.b_off), tk.k, n,
                             sign_mask(tk.sign), row, col);
  }
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int r = r0 + 8 * i + lr, c = c0 + 4 * j + lc;
      if (r < m && c < n) C[cb.c_off + (int64_t)r * n + c] = acc[i][j];
    }
}

// The tile at (r0, c0), as wide as the block leaves it (up to kF64TileCols columns).
template <typename T, int TM>
__device__ __forceinline__ void f64_tile_cols(const GemmCBlk& cb, const GemmTask* __restrict__ task, int r0, int c0,
                                              int lane, const T* __restrict__ A, const T* __restrict__ As,
                                              const T* __restrict__ B, const T* __restrict__ Bs, T* __restrict__ C) {
  const int n = cb.n - c0;
  if (n > 12) f64_tile<T, TM, 4>(cb, task, r0, c0, lane, A, As, B, Bs, C);
  else if (n > 8) f64_tile<T, TM, 3>(cb, task, r0, c0, lane, A, As, B, Bs, C);
  else if (n > 4) f64_tile<T, TM, 2>(cb, task, r0, c0, lane, A, As, B, Bs, C);
  else f64_tile<T, TM, 1>(cb, task, r0, c0, lane, A, As, B, Bs, C);
}

// Output tiles of 8 TM x 16. The FP64 pipe takes about 20 SM cycles per warp instruction and
// each of the four sub-partitions has its own quarter of it, so what decides this kernel is how
// evenly the multiply-adds spread over the sub-partitions and how few of them are padding;
// operand reads are cheap beside that. Hence a warp owns a tile (no CTA-wide barrier), a tile at a
// block's edge is run at the size of the 8 x 4 pieces that hold outputs (at most 7 rows and 3
// columns of padding), and tiles are taken longest-first from an atomic counter (zeroed before
// the launch). One warp alone needs 320 cycles per k; where that makes the longest tile too long
// for the launch (share_tiles), a CTA's four warps share each tile, four columns each.
// Measured (D = 4000 matvec steps 0 and 3): 2.44 and 2.45 ms = 1.07 of cuBLAS DGEMM's 1.1
// TFLOP/s, against 2.91 and 3.19 ms for 32 x 32 tiles of a CTA staged in shared memory, and 2.52
// and 2.58 ms with the pieces outside a block predicated off; D = 1000: 231 and 252 us against
// 318 and 392 us (launch, transposes and skinny blocks included).
template <typename T, int TM, bool SHARE>
__global__ void __launch_bounds__(NT, sizeof(T) == 8 ? (TM == 1 ? 4 : 3) : 2) k_gemm_f64(const GemmCBlk* __restrict__ cblk, const GemmTask* __restrict__ task,
                                                 const GemmTileRun* __restrict__ runs, int nruns, int ntiles,
                                                 const T* __restrict__ A, const T* __restrict__ As,
                                                 const T* __restrict__ B, const T* __restrict__ Bs,
                                                 T* __restrict__ C, int* __restrict__ counter) {
  static_assert(NT / 32 == kF64TileCols / 4, "a shared tile has one piece column per warp");
  __shared__ int s_ti;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  while (true) {
    int ti = 0;
    if (SHARE) {
      __syncthreads();   // everyone has read s_ti
      if (threadIdx.x == 0) s_ti = atomicAdd(counter, 1);
      __syncthreads();
      ti = s_ti;
    } else {
      if (lane == 0) ti = atomicAdd(counter, 1);
      ti = __shfl_sync(0xffffffffu, ti, 0);
    }
    if (ti >= ntiles) break;
    int lo = 0, hi = nruns - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (__ldg(&runs[mid].begin) <= ti) lo = mid; else hi = mid - 1;
    }
    const GemmTileRun run = runs[lo];
    const GemmCBlk cb = cblk[run.cblk];
    const int l = ti - run.begin, lm = l / run.tn_count;
    const int r0 = (run.tm0 + lm) * (8 * TM), c0 = (run.tn0 + l - lm * run.tn_count) * kF64TileCols;
    if constexpr (SHARE) {
      if (c0 + 4 * warp >= cb.n) continue;
      if (TM > 1 && r0 + 8 >= cb.m) f64_tile<T, 1, 1>(cb, task, r0, c0 + 4 * warp, lane, A, As, B, Bs, C);
      else f64_tile<T, TM, 1>(cb, task, r0, c0 + 4 * warp, lane, A, As, B, Bs, C);
    } else if (TM > 1 && r0 + 8 >= cb.m) {
      f64_tile_cols<T, 1>(cb, task, r0, c0, lane, A, As, B, Bs, C);
    } else {
      f64_tile_cols<T, TM>(cb, task, r0, c0, lane, A, As, B, Bs, C);
    }
  }
}

// Skinny output blocks (n <= 8, every task k <= 8). An FP64 instruction costs the same whatever
// lanes are active, so a block's m x n outputs are taken as one flat range, one per lane and up to
// four ranges of 32 at once: every lane has an output whatever m and n are, and the stores are
// contiguous. Operand reads are cheap beside that (lanes of one row share an address). The block's
// entries (its tasks' k values end to end) are worked off kSkinnyDepth at a time: their records,
// then all their A and B values, then the multiply-adds, so a pass waits about twice for memory
// and not twice per task; the next pass's record is read ahead. Bound by the FP64 pipe where a
// launch has enough passes, else by those waits.
// Measured against one thread per row (256 rows per CTA, n columns in registers): MPO part of the
// D = 4000 matvec 126 -> 118 us (114 us of multiply-adds at the pipe's rate), the two MPO steps of
// the D = 3000 complex Hubbard matvec 245 -> 145 us, its blocks of a few rows 171 -> 64 us. Depth 1
// / 2 / 3 / 4: 401 / 390 / 393 / 399 us per D = 4000 matvec.
constexpr int kSkinnyThreads = 128;
constexpr int kSkinnyMax = 8;
constexpr int kSkinnyPass = 128;   // outputs of one pass
constexpr int kSkinnyDepth = 2;

// Scale field of an output value as the split path defines it (0 for zero, else
// max(1, biased exponent)); complex outputs are never folded.
__device__ __forceinline__ int out_field(double v) {
  const uint32_t hi = (uint32_t)__double2hiint(v) & 0x7FFFFFFFu, lo = (uint32_t)__double2loint(v);
  return (hi | lo) ? max(1, (int)(hi >> 20)) : 0;
}
__device__ __forceinline__ int out_field(double2 v) { return max(out_field(v.x), out_field(v.y)); }

// atomicMax of v into fields[key] once per group of lanes with the same key.
__device__ __forceinline__ void fold_field(unsigned mask, int key, int v, int32_t* __restrict__ fields) {
  const unsigned m = __match_any_sync(mask, key);
  const int x = (int)__reduce_max_sync(m, (unsigned)max(v, 0));
  if (key >= 0 && x > 0 && (int)(threadIdx.x & 31) == __ffs(m) - 1) atomicMax(fields + key, x);
}

// Outputs o + lane + 32 u (u < U, clamped into the block) of one block, from all its entries. I: the
// type of an output's position in its block.
template <typename T, typename I, int U>
__device__ __forceinline__ void skinny_pass(const GemmCBlk& cb, const SkinnyItem& item, I o, int lane,
                                            const SkinnyEntry* __restrict__ entry, const T* __restrict__ A,
                                            const T* __restrict__ As, const T* __restrict__ B, const T* __restrict__ Bs,
                                            T* __restrict__ C, const SkinnyFuse& fz, int32_t* __restrict__ fields) {
  const I total = (I)cb.m * cb.n;
  int row[U], col[U];
  T acc[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const I x = min(o + 32 * u + lane, total - 1);
    row[u] = (int)(x / cb.n);
    col[u] = (int)(x - (I)row[u] * cb.n);
    acc[u] = zero_of(T());
  }
  int e = item.e0;
  for (; e + kSkinnyDepth <= item.e1; e += kSkinnyDepth) {
    T av[kSkinnyDepth][U], bv[kSkinnyDepth][U];
#pragma unroll
    for (int t = 0; t < kSkinnyDepth; ++t) {
      const SkinnyEntry x = entry[e + t];
      const T* a = operand_block(A, As, x.a_off);
      const T* b = operand_block(B, Bs, x.b_off);
      const unsigned long long sg = sign_mask(x.sign);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        av[t][u] = flip(__ldg(a + (int64_t)row[u] * x.a_rs), sg);
        bv[t][u] = __ldg(b + col[u]);
      }
    }
#pragma unroll
    for (int t = 0; t < kSkinnyDepth; ++t)
#pragma unroll
      for (int u = 0; u < U; ++u) fma_acc(acc[u], av[t][u], bv[t][u]);
  }
#pragma unroll 1
  for (; e < item.e1; ++e) {   // a loop: predicated-off multiply-adds would cost as much as executed ones
    const SkinnyEntry x = entry[e];
    const T* a = operand_block(A, As, x.a_off);
    const T* b = operand_block(B, Bs, x.b_off);
    const unsigned long long sg = sign_mask(x.sign);
#pragma unroll
    for (int u = 0; u < U; ++u) fma_acc(acc[u], flip(__ldg(a + (int64_t)row[u] * x.a_rs), sg), __ldg(b + col[u]));
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const I x = o + 32 * u + lane;
    if (x < total) C[cb.c_off + x] = acc[u];
    // the outputs' order is that of the later operand's rows of k3 values
    if (fz.exp_base >= 0) fold_field(0xffffffffu, x < total ? fz.exp_base + (int)(x / fz.k3) : -1, out_field(acc[u]), fields);
  }
}

// I = int64_t where a block has 2^31 outputs or more (17 GB of FP64 values); 64-bit divisions would
// cost the others.
template <typename T, typename I>
__global__ void __launch_bounds__(kSkinnyThreads, sizeof(T) == 8 ? 7 : 5) k_gemm_skinny(
    const GemmCBlk* __restrict__ cblk, const SkinnyEntry* __restrict__ entry, const SkinnyItem* __restrict__ items,
    int npasses, int shift, const T* __restrict__ A, const T* __restrict__ As, const T* __restrict__ B,
    const T* __restrict__ Bs, T* __restrict__ C, const SkinnyFuse* __restrict__ fuse, int32_t* __restrict__ fields) {
  const int lane = threadIdx.x & 31, step = gridDim.x * (kSkinnyThreads / 32);
  int it = blockIdx.x * (kSkinnyThreads / 32) + (threadIdx.x >> 5);
  if (it >= npasses) return;
  SkinnyItem next = items[it >> shift];
  for (; it < npasses; it += step) {
    const SkinnyItem item = next;
    const I o = (I)(item.p0 + (it & ((1 << shift) - 1))) * kSkinnyPass;
    if (it + step < npasses) next = items[(it + step) >> shift];
    const GemmCBlk cb = cblk[item.cblk];
    const I left = (I)cb.m * cb.n - o;
    if (left <= 0) continue;
    const SkinnyFuse fz = fuse ? fuse[item.cblk] : SkinnyFuse{-1, 1};
    if (left > 96) skinny_pass<T, I, 4>(cb, item, o, lane, entry, A, As, B, Bs, C, fz, fields);
    else if (left > 64) skinny_pass<T, I, 3>(cb, item, o, lane, entry, A, As, B, Bs, C, fz, fields);
    else if (left > 32) skinny_pass<T, I, 2>(cb, item, o, lane, entry, A, As, B, Bs, C, fz, fields);
    else skinny_pass<T, I, 1>(cb, item, o, lane, entry, A, As, B, Bs, C, fz, fields);
  }
}

}  // namespace

bool skinny_cblk(const GemmSchedule& g, int32_t q) {
  const GemmCBlk& cb = g.cblk[q];
  if (cb.n > kSkinnyMax) return false;
  for (int32_t t = cb.t0; t < cb.t1; ++t)
    if (g.task[t].k > kSkinnyMax) return false;
  return true;
}

template <typename T, typename I>
void launch_skinny(const GemmSchedule& g, const Operands& op, void* c, int grid, cudaStream_t s, const SkinnyFuse* fuse,
                   int32_t* fields) {
  const int shift = g.skinny_outputs == 4 * kSkinnyPass ? 2 : 0;
  k_gemm_skinny<T, I><<<grid, kSkinnyThreads, 0, s>>>(
      g.d_cblk.as<GemmCBlk>(), g.d_entry.as<SkinnyEntry>(), g.d_skinny.as<SkinnyItem>(), (int)g.skinny.size() << shift,
      shift, static_cast<const T*>(op.a), static_cast<const T*>(op.a_src), static_cast<const T*>(op.b),
      static_cast<const T*>(op.b_src), static_cast<T*>(c), fuse, fields);
}

template <typename T, int TM, bool SHARE>
void launch_f64_t(const GemmSchedule& g, const Operands& op, void* c, int num_sms, cudaStream_t s) {
  const int64_t per_cta = SHARE ? 1 : NT / 32;
  const int grid = (int)std::min<int64_t>((g.ntiles + per_cta - 1) / per_cta, (int64_t)std::max(1, num_sms) * kF64CtasPerSm);
  k_gemm_f64<T, TM, SHARE><<<grid, NT, 0, s>>>(
      g.d_cblk.as<GemmCBlk>(), g.d_task.as<GemmTask>(), g.d_run.as<GemmTileRun>(), (int)g.run.size(), (int)g.ntiles,
      static_cast<const T*>(op.a), static_cast<const T*>(op.a_src), static_cast<const T*>(op.b),
      static_cast<const T*>(op.b_src), static_cast<T*>(c), g.d_counter.as<int>());
}

template <typename T>
void launch_f64(const GemmSchedule& g, const Operands& op, void* c, int num_sms, cudaStream_t s) {
  if (g.bm == 64) {
    if (g.share_tiles) launch_f64_t<T, 2, true>(g, op, c, num_sms, s);
    else launch_f64_t<T, 2, false>(g, op, c, num_sms, s);
  } else {
    if (g.share_tiles) launch_f64_t<T, 1, true>(g, op, c, num_sms, s);
    else launch_f64_t<T, 1, false>(g, op, c, num_sms, s);
  }
}

// CTAs of one full wave.
template <typename T>
int skinny_wave(int num_sms) {
  static int per_sm = [] {
    int n = 0;
    QLTG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_gemm_skinny<T, int32_t>, kSkinnyThreads, 0));
    return std::max(1, n);
  }();
  return std::max(1, num_sms) * per_sm;
}

int skinny_grid(int items, bool cplx, int num_sms) {
  // Complex: up to four waves. An equal share of passes per warp is not an equal share of work
  // (their entries differ), and with one wave the SMs finish up to a sixth apart: Hubbard MPO steps
  // 71 / 75 -> 62 / 69 us. The real passes are four times shorter and the start of a CTA weighs
  // more: D = 4000 MPO 120 us with one wave, 122 with four.
  const int wave = cplx ? 4 * skinny_wave<double2>(num_sms) : skinny_wave<double>(num_sms);
  const int per_cta = kSkinnyThreads / 32;
  return std::max(1, std::min((items + per_cta - 1) / per_cta, wave));
}

void launch_gemm_f64_skinny(const GemmSchedule& g, const Operands& op, void* c, bool cplx, int num_sms,
                            cudaStream_t s, const SkinnyFuse* fuse, int32_t* fields) {
  const int ns = (int)g.skinny.size();
  if (!ns) return;
  const int grid = skinny_grid(ns, cplx, num_sms);
  auto* launch = g.skinny_long ? (cplx ? launch_skinny<double2, int64_t> : launch_skinny<double, int64_t>)
                               : (cplx ? launch_skinny<double2, int32_t> : launch_skinny<double, int32_t>);
  launch(g, op, c, grid, s, fuse, fields);
  QLTG_CUDA(cudaGetLastError());
}

void launch_gemm_f64(const GemmSchedule& g, const Operands& op, void* c, bool cplx, int num_sms, cudaStream_t s) {
  launch_gemm_f64_skinny(g, op, c, cplx, num_sms, s);
  if (!g.ntiles) return;
  QLTG_CUDA(cudaMemsetAsync(g.d_counter.get(), 0, sizeof(int), s));
  if (cplx) launch_f64<double2>(g, op, c, num_sms, s);
  else launch_f64<double>(g, op, c, num_sms, s);
  QLTG_CUDA(cudaGetLastError());
}

// ------------------------------------------------------------------ FP64 rate self-test
// The two FP64 arithmetic paths of this GPU side by side, measured rather than assumed: a
// DFMA loop (8 independent chains per thread) and an mma.sync m8n8k4 f64 loop (4 independent
// accumulator fragments per warp; 8 x 8 x 4 multiply-adds = 512 flops per instruction). The
// FP64 GEMM kernels above use DFMA because the two run at the same rate here while the MMA
// path pads every block to 8 x 8 x 4 fragments.
constexpr int kRateIters = 4096;
__global__ void __launch_bounds__(256) k_rate_dfma(double* out, double seed) {
  double a[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) a[i] = seed + threadIdx.x + i;
  const double b = 1.0 + 1e-12 * seed, c = 1e-300;
  for (int it = 0; it < kRateIters; ++it)
#pragma unroll
    for (int i = 0; i < 8; ++i) a[i] = fma(a[i], b, c);
  double t = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) t += a[i];
  if (t == 1.2345) out[0] = t;   // keeps the loop; never true for these inputs
}
__global__ void __launch_bounds__(256) k_rate_dmma(double* out, double seed) {
  const double av = seed + (threadIdx.x & 31), bv = 1.0 + 1e-12 * seed;
  double d[4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i) d[i][0] = d[i][1] = 0.0;
  for (int it = 0; it < kRateIters; ++it)
#pragma unroll
    for (int i = 0; i < 4; ++i)
      asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                   : "+d"(d[i][0]), "+d"(d[i][1])
                   : "d"(av), "d"(bv));
  double t = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) t += d[i][0] + d[i][1];
  if (t == 1.2345) out[0] = t;
}

void fp64_rates(int num_sms, cudaStream_t s, double* dfma_tflops, double* dmma_tflops) {
  DevBuf sink(sizeof(double));
  const int grid = std::max(1, num_sms) * 8;
  cudaEvent_t e[4];
  for (auto& x : e) QLTG_CUDA(cudaEventCreate(&x));
  k_rate_dfma<<<grid, 256, 0, s>>>(sink.as<double>(), 1.0);   // warm-up
  k_rate_dmma<<<grid, 256, 0, s>>>(sink.as<double>(), 1.0);
  QLTG_CUDA(cudaEventRecord(e[0], s));
  k_rate_dfma<<<grid, 256, 0, s>>>(sink.as<double>(), 2.0);
  QLTG_CUDA(cudaEventRecord(e[1], s));
  QLTG_CUDA(cudaEventRecord(e[2], s));
  k_rate_dmma<<<grid, 256, 0, s>>>(sink.as<double>(), 2.0);
  QLTG_CUDA(cudaEventRecord(e[3], s));
  QLTG_CUDA(cudaGetLastError());
  QLTG_CUDA(cudaEventSynchronize(e[3]));
  float ms_f = 0, ms_m = 0;
  QLTG_CUDA(cudaEventElapsedTime(&ms_f, e[0], e[1]));
  QLTG_CUDA(cudaEventElapsedTime(&ms_m, e[2], e[3]));
  for (auto x : e) cudaEventDestroy(x);
  const double threads = (double)grid * 256, warps = threads / 32;
  *dfma_tflops = threads * kRateIters * 8 * 2 / (ms_f * 1e-3) / 1e12;
  *dmma_tflops = warps * kRateIters * 4 * 512 / (ms_m * 1e-3) / 1e12;
}

}  // namespace qltg
