// Batched block permutation: one launch permutes every block of a tensor.
//
// Replaces the reference's per-block hp_numeric::TensorTranspose (HPTT plan + execute on
// the CPU, a cuTENSOR plan / permute / destroy per block on the GPU;
// framework/hp_numeric/ten_trans.h:56-114, :245-349) and the ±1 block sign of
// BlockSparseDataTensor::Transpose (global_operations.h:393-441).
//
// Per block, unit dims are squeezed and destination-adjacent dims that are also adjacent in the
// source are merged. What is left is cut into work items of one warp each (8 KB of data), which
// need no CTA-wide barrier and have all their loads in flight at once, 20 warps per SM:
//  * tile: a box over the source-inner dims P (one, or two when the first is short) and the
//    destination-inner dims Q (likewise), about 32 x 32, read along P and written along Q through
//    shared memory (rows an odd number of elements apart: no bank conflicts). Two dims on a side
//    keep the runs long when the innermost extent is 3 (an MPO bond): P and Q index ranges are
//    contiguous in the source and in the destination;
//  * whole: a block of up to 8 KB that no single tile covers, read and written as one flat range;
//  * runs: the innermost dim is the same on both sides, so runs (or pieces of long ones) are
//    copied, a flat range of as many runs as make 8 KB.
// The +-1 block sign is applied by flipping the sign bit (no floating-point multiply). Bound by
// HBM: lenv . psi at D = 4000 (80 MB) reversed 32.9 us = 0.71 of the measured copy rate, 107 us
// with CTA-wide tiles of power-of-two extents; the 5544 blocks of a complex Hubbard psi (20 MB,
// from L2) 8.2 us, 57 us before - there the descriptor and data latencies of one item bound it.
#include <algorithm>
#include <string>
#include <tuple>

#include "ctrct.h"

namespace qltg {
namespace {

constexpr int kPermWarps = 4;      // per CTA
constexpr int kPermThreads = 32 * kPermWarps;
constexpr int kPermCtasPerSm = 5;   // 3 / 4 / 5 / 6 / 8 (smaller tiles): 34.8 / 32.9 / 32.9 / 38.7 / 41.2 us at D = 4000 (below)
// Elements of one warp's buffer: 32 rows of 33 FP64 values, or as many bytes of complex ones.
// Small enough that division by an extent is a multiplication (see inv_of).
__host__ __device__ constexpr int perm_cap(int elem_bytes) { return elem_bytes == 16 ? 528 : 1056; }

__device__ __forceinline__ double flip(double x, uint64_t m) {
  return __longlong_as_double(__double_as_longlong(x) ^ (long long)m);
}
__device__ __forceinline__ double2 flip(double2 x, uint64_t m) { return make_double2(flip(x.x, m), flip(x.y, m)); }

// e / d for e, d <= 1056 (the largest buffer) as (e inv_of(d)) >> 21: the product is below 2^32, and
// rounding the reciprocal up adds less than e / 2^21 to the quotient, which is below 1 / d.
__host__ __device__ __forceinline__ uint32_t inv_of(uint32_t d) { return ((1u << 21) + d - 1) / d; }
__device__ __forceinline__ uint32_t div_by(uint32_t e, uint32_t inv) { return (e * inv) >> 21; }

// Source and destination offsets of index `rem` over the descriptor's dims (last fastest).
__device__ __forceinline__ void outer_offsets(const PermDesc& d, uint32_t rem, uint32_t& soff, uint32_t& doff) {
  soff = doff = 0;
  for (int i = d.nd - 1; i >= 0; --i) {
    const uint32_t di = d.dims[i], q = rem / di, x = rem - q * di;
    rem = q;
    soff += x * d.sstr[i];
    doff += x * d.dstr[i];
  }
}

template <typename T>
__device__ __forceinline__ void cp_async_elem(T* dst, const T* src) {
  if constexpr (sizeof(T) == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
  else
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <typename T>
__global__ void __launch_bounds__(kPermThreads, kPermCtasPerSm) k_permute(const PermDesc* __restrict__ descs, int nd,
                                                          const int32_t* __restrict__ item_block, int64_t nitems,
                                                          const T* __restrict__ src, T* __restrict__ dst) {
  constexpr int kCap = perm_cap((int)sizeof(T));
  constexpr int kBatch = 8;   // loads in flight per lane of a copy
  __shared__ __align__(16) T s_buf[kPermWarps][kCap];
  const int warp = threadIdx.x >> 5;
  const uint32_t lane = threadIdx.x & 31;
  T* S = s_buf[warp];
  const int64_t first = (int64_t)blockIdx.x * kPermWarps + warp, step = (int64_t)gridDim.x * kPermWarps;
  int next = item_block && first < nitems ? __ldg(item_block + first) : 0;
  for (int64_t item = first; item < nitems; item += step) {
    int b = next;
    if (item_block) {
      // the next item's descriptor is on its way while this one is worked on
      if (item + step < nitems) {
        next = __ldg(item_block + item + step);
        if (lane < (sizeof(PermDesc) + 127) / 128)
          asm volatile("prefetch.global.L1 [%0];" ::"l"(reinterpret_cast<const char*>(descs + next) + min(lane * 128, (uint32_t)sizeof(PermDesc) - 1)));
      }
    } else {
      int hi = nd - 1;
      b = 0;
      while (b < hi) {
        const int mid = (b + hi + 1) >> 1;
        if (descs[mid].tile_begin <= item) b = mid; else hi = mid - 1;
      }
    }
    const PermDesc& d = descs[b];
    const uint32_t local = (uint32_t)(item - d.tile_begin);
    const uint64_t sg = d.sign_mask;
    const T* s = src + d.src_off;
    T* o = dst + d.dst_off;
    if (d.mode == kPermTile) {
      // the tile's place: p0, p1, q0, q1 tiles, then the outer index
      uint32_t rem = local, t0 = d.tp[0], t1 = d.tp[1], t2 = d.tq[0], t3 = d.tq[1];
      uint32_t x = rem / t0;
      const uint32_t p0 = (rem - x * t0) * d.ep[0];
      rem = x; x = rem / t1;
      const uint32_t p1 = (rem - x * t1) * d.ep[1];
      rem = x; x = rem / t2;
      const uint32_t q0 = (rem - x * t2) * d.eq[0];
      rem = x; x = rem / t3;
      const uint32_t q1 = (rem - x * t3) * d.eq[1];
      uint32_t soff, doff;
      outer_offsets(d, x, soff, doff);
      const uint32_t wp0 = min(d.ep[0], d.np[0] - p0), wp1 = min(d.ep[1], d.np[1] - p1);
      const uint32_t wq0 = min(d.eq[0], d.nq[0] - q0), wq1 = min(d.eq[1], d.nq[1] - q1);
      const uint32_t wp = wp0 * wp1, wq = wq0 * wq1, n = wp * wq, pitch = wp | 1;
      const uint32_t sq0 = d.sq[0], sq1 = d.sq[1], dp0 = d.dp[0], dp1 = d.dp[1];
      // p1 (q1) tiles hold all of p0 (q0), so P (Q) is one contiguous range of the source (destination)
      s += soff + p0 + p1 * d.np[0] + q0 * sq0 + q1 * sq1;
      o += doff + q0 + q1 * d.nq[0] + p0 * dp0 + p1 * dp1;
      // A side of 17 .. 32 goes one lane per index, the other side's offset carried along; any
      // other extent as one flat range, divided by its extents.
      if (wp > 16 && wp <= 32) {
        if (lane < wp) {
          const T* row = s + lane;
          T* at = S + lane;
          const uint32_t wrap = sq1 - wq0 * sq0;
          uint32_t y0 = 0;
#pragma unroll 8
          for (uint32_t q = 0; q < wq; ++q) {
            cp_async_elem(at, row);
            at += pitch;
            row += sq0;
            if (++y0 == wq0) {
              y0 = 0;
              row += (int32_t)wrap;
            }
          }
        }
      } else {
        const uint32_t iwp = inv_of(wp), iwq0 = inv_of(wq0);
#pragma unroll 4
        for (uint32_t e = lane; e < n; e += 32) {
          const uint32_t q = div_by(e, iwp), p = e - q * wp, y1 = div_by(q, iwq0), y0 = q - y1 * wq0;
          cp_async_elem(S + q * pitch + p, s + (y0 * sq0 + y1 * sq1 + p));
        }
      }
      cp_async_wait_all();
      __syncwarp();
      if (wq > 16 && wq <= 32) {
        if (lane < wq) {
          T* row = o + lane;
          const T* at = S + lane * pitch;
          const uint32_t wrap = dp1 - wp0 * dp0;
          uint32_t x0 = 0;
#pragma unroll 8
          for (uint32_t p = 0; p < wp; ++p) {
            *row = flip(at[p], sg);
            row += dp0;
            if (++x0 == wp0) {
              x0 = 0;
              row += (int32_t)wrap;
            }
          }
        }
      } else {
        const uint32_t iwq = inv_of(wq), iwp0 = inv_of(wp0);
#pragma unroll 4
        for (uint32_t e = lane; e < n; e += 32) {
          const uint32_t p = div_by(e, iwq), q = e - p * wq, x1 = div_by(p, iwp0), x0 = p - x1 * wp0;
          o[x0 * dp0 + x1 * dp1 + q] = flip(S[q * pitch + p], sg);
        }
      }
    } else if (d.mode == kPermWhole) {
      const uint32_t n = d.size;
#pragma unroll 4
      for (uint32_t e = lane; e < n; e += 32) cp_async_elem(S + e, s + e);
      cp_async_wait_all();
      __syncwarp();
      for (uint32_t e = lane; e < n; e += 32) {
        uint32_t rem = e, at = 0;
        for (int i = d.nd - 1; i >= 0; --i) {
          const uint32_t x = div_by(rem, d.dstr[i]);   // here the dims' reciprocals
          at += (rem - x * d.dims[i]) * d.sstr[i];
          rem = x;
        }
        o[e] = flip(S[at], sg);
      }
    } else if (d.per > 1) {
      // runs run0 .. run0 + nr - 1, their offsets once (one lane per run) into the buffer
      const uint32_t len = d.size, run0 = local * d.per;
      uint32_t runs = 1;
      for (int i = 0; i < d.nd; ++i) runs *= d.dims[i];
      const uint32_t nr = min(d.per, runs - run0), n = nr * len, inv = inv_of(len);
      uint2* off = reinterpret_cast<uint2*>(S);
      for (uint32_t r = lane; r < nr; r += 32) outer_offsets(d, run0 + r, off[r].x, off[r].y);
      __syncwarp();
      for (uint32_t e0 = lane; e0 < n; e0 += 32 * kBatch) {
        T v[kBatch];
        uint32_t at[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
          const uint32_t e = e0 + 32 * u;
          if (e < n) {
            const uint32_t r = div_by(e, inv), x = e - r * len;
            const uint2 f = off[r];
            v[u] = __ldg(s + (f.x + x));
            at[u] = f.y + x;
          }
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u)
          if (e0 + 32 * u < n) o[at[u]] = flip(v[u], sg);
      }
    } else {
      // a piece of a long run
      const uint32_t len = d.size, chunk = (uint32_t)kCap & ~31u, pieces = (len + chunk - 1) / chunk, run = local / pieces;
      const uint32_t c0 = (local - run * pieces) * chunk, n = min(chunk, len - c0);
      uint32_t soff, doff;
      outer_offsets(d, run, soff, doff);
      s += soff + c0;
      o += doff + c0;
      for (uint32_t e0 = lane; e0 < n; e0 += 32 * kBatch) {
        T v[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u)
          if (e0 + 32 * u < n) v[u] = __ldg(s + e0 + 32 * u);
#pragma unroll
        for (int u = 0; u < kBatch; ++u)
          if (e0 + 32 * u < n) o[e0 + 32 * u] = flip(v[u], sg);
      }
    }
    __syncwarp();   // the buffer is free again
  }
}

// Items of one block; fills the descriptor's mode and shape from its squeezed dims in destination
// order (extents dd, source strides ds, innermost last).
int64_t plan_block(PermDesc& d, int m, const int64_t* dd, const int64_t* ds, int elem_bytes) {
  const int cap = perm_cap(elem_bytes);
  int64_t total = 1, dstr[kMaxRank];
  for (int i = m - 1; i >= 0; --i) {
    dstr[i] = total;
    total *= dd[i];
  }
  auto keep = [&](int i) {   // dim i joins the descriptor's list
    d.dims[d.nd] = (uint32_t)dd[i];
    d.sstr[d.nd] = (uint32_t)ds[i];
    d.dstr[d.nd] = (uint32_t)dstr[i];
    ++d.nd;
  };
  int p = -1;
  for (int i = 0; i < m; ++i)
    if (ds[i] == 1) p = i;
  if (m == 0 || p == m - 1) {
    // runs; a small block is one flat item either way
    d.mode = kPermRuns;
    const int64_t len = m ? dd[m - 1] : 1, runs = total / len;
    for (int i = 0; i < m - 1; ++i) keep(i);
    d.size = (uint32_t)len;
    if (2 * len <= cap && runs > 1) {
      // as many runs as the buffer has room for their data; their offsets (8 bytes each) fit then too
      d.per = (uint32_t)std::max<int64_t>(2, cap / len);
      return (runs + d.per - 1) / d.per;
    }
    d.per = 1;
    const int64_t chunk = cap & ~31;
    return runs * ((len + chunk - 1) / chunk);
  }
  // tile: q0 = the innermost destination dim, p0 = the innermost source dim; a short one takes
  // its neighbour as a second dim
  constexpr int kShort = 16;
  const int q0 = m - 1;
  int q1 = -1, p1 = -1;
  if (dd[q0] <= kShort && m - 2 != p) q1 = m - 2;
  if (dd[p] <= kShort)
    for (int i = 0; i < m; ++i)
      if (ds[i] == dd[p] && i != q0 && i != q1) p1 = i;
  const int side = elem_bytes == 16 ? 22 : 32;
  int64_t np[2] = {dd[p], p1 >= 0 ? dd[p1] : 1}, nq[2] = {dd[q0], q1 >= 0 ? dd[q1] : 1}, ep[2], eq[2];
  auto start = [&](const int64_t* n, int64_t* e, bool two) {
    e[0] = two ? n[0] : std::min<int64_t>(n[0], side);
    e[1] = two ? std::min<int64_t>(n[1], std::max<int64_t>(1, side / n[0])) : 1;
  };
  start(np, ep, p1 >= 0);
  start(nq, eq, q1 >= 0);
  // grow the side that can while the tile leaves half the buffer unused
  auto fits = [&](int64_t a0, int64_t a1, int64_t b0, int64_t b1) { return ((a0 * a1) | 1) * b0 * b1 <= cap; };
  for (bool grown = true; grown;) {
    grown = false;
    int64_t& gp = p1 >= 0 ? ep[1] : ep[0];
    int64_t& gq = q1 >= 0 ? eq[1] : eq[0];
    const int64_t lp = p1 >= 0 ? np[1] : np[0], lq = q1 >= 0 ? nq[1] : nq[0];
    for (int side_no = 0; side_no < 2 && !grown; ++side_no) {
      int64_t& g = side_no == 0 ? gp : gq;
      const int64_t l = side_no == 0 ? lp : lq, was = g;
      if (g >= l) continue;
      g = std::min(l, 2 * g);
      if (fits(ep[0], ep[1], eq[0], eq[1])) grown = true;
      else g = was;
    }
  }
  int64_t outer = total, tiles = 1;
  for (int i = 0; i < 2; ++i) {
    for (auto [n, e, t] : {std::tuple<int64_t*, int64_t*, uint32_t*>{&np[i], &ep[i], &d.tp[i]}, {&nq[i], &eq[i], &d.tq[i]}}) {
      const int64_t cnt = (*n + *e - 1) / *e;
      *e = (*n + cnt - 1) / cnt;   // even pieces
      *t = (uint32_t)((*n + *e - 1) / *e);
      tiles *= *t;
      outer /= *n;
    }
    d.np[i] = (uint32_t)np[i];
    d.ep[i] = (uint32_t)ep[i];
    d.nq[i] = (uint32_t)nq[i];
    d.eq[i] = (uint32_t)eq[i];
  }
  if (outer > 1 && total <= cap) {
    d.mode = kPermWhole;
    for (int i = 0; i < m; ++i) {
      keep(i);
      d.dstr[i] = inv_of((uint32_t)dd[i]);
    }
    d.size = (uint32_t)total;
    return 1;
  }
  d.mode = kPermTile;
  d.dp[0] = (uint32_t)dstr[p];
  d.dp[1] = p1 >= 0 ? (uint32_t)dstr[p1] : 0;
  d.sq[0] = (uint32_t)ds[q0];
  d.sq[1] = q1 >= 0 ? (uint32_t)ds[q1] : 0;
  for (int i = 0; i < m; ++i)
    if (i != p && i != p1 && i != q0 && i != q1) keep(i);
  return tiles * outer;
}

template <typename T>
void launch_permute(const PermDesc* descs, int64_t nblocks, const int32_t* item_block, int64_t nitems, const void* src,
                    void* dst, cudaStream_t s) {
  check_aligned(sizeof(T), {src, dst});
  const unsigned grid = (unsigned)std::min<int64_t>((nitems + kPermWarps - 1) / kPermWarps,
                                                    (int64_t)current_sm_count() * kPermCtasPerSm);
  k_permute<T><<<grid, kPermThreads, 0, s>>>(descs, (int)nblocks, item_block, nitems, static_cast<const T*>(src),
                                             static_cast<T*>(dst));
  QLTG_CUDA(cudaGetLastError());
}

}  // namespace

void TransposeList::describe(const Meta& t, const std::vector<int>& order, const std::vector<double>& signs,
                             const std::vector<int64_t>* dst_offsets, bool skip_identity,
                             const std::vector<uint8_t>* skip) {
  host.clear();
  host.reserve(t.nblk);
  identity.assign(t.nblk, 0);
  ntiles = 0;
  const int r = t.rank;
  for (int64_t b = 0; b < t.nblk; ++b) {
    PermDesc d{};
    d.src_off = t.offsets[b];
    d.dst_off = dst_offsets ? (*dst_offsets)[b] : t.offsets[b];
    d.sign_mask = (!signs.empty() && signs[b] < 0) ? 0x8000000000000000ull : 0ull;
    int64_t sstr[kMaxRank];
    sstr[r - 1] = 1;
    for (int i = r - 2; i >= 0; --i) sstr[i] = sstr[i + 1] * t.dim(b, i + 1);
    // destination-order dims / strides, unit dims dropped
    int64_t dd[kMaxRank], ds[kMaxRank];
    int n = 0;
    for (int i = 0; i < r; ++i) {
      const int64_t dim = t.dim(b, order[i]);
      if (dim == 1) continue;
      dd[n] = dim;
      ds[n] = sstr[order[i]];
      ++n;
    }
    // merge destination neighbours that are source neighbours in the same order
    int m = 0;
    for (int i = 0; i < n; ++i) {
      if (m > 0 && ds[m - 1] == ds[i] * dd[i]) {
        dd[m - 1] *= dd[i];
        ds[m - 1] = ds[i];
      } else {
        dd[m] = dd[i];
        ds[m] = ds[i];
        ++m;
      }
    }
    for (int i = 0; i < m; ++i) QLTG_CHECK(dd[i] < ((int64_t)1 << 31), QLTG_ERR_UNSUPPORTED, "block dimension above 2^31");
    QLTG_CHECK(t.blk_size(b) < ((int64_t)1 << 31), QLTG_ERR_UNSUPPORTED, "block with 2^31 or more elements");
    // at most one non-unit dim left after merging: the block's data is laid out the same way
    identity[b] = m <= 1 && d.sign_mask == 0 && d.src_off == d.dst_off;
    const bool none = (identity[b] && skip_identity) || (skip && (*skip)[b]);
    const int64_t tiles = none ? 0 : plan_block(d, m, dd, ds, (int)t.elem_bytes());
    d.tile_begin = ntiles;
    ntiles += tiles;
    host.push_back(d);
  }
  nblocks = (int64_t)host.size();
}

void TransposeList::build(const Meta& t, const std::vector<int>& order, const std::vector<double>& signs,
                          const std::vector<int64_t>* dst_offsets, cudaStream_t s, bool skip_identity,
                          const std::vector<uint8_t>* skip) {
  describe(t, order, signs, dst_offsets, skip_identity, skip);
  QLTG_CHECK(ntiles < ((int64_t)1 << 32) && nblocks < ((int64_t)1 << 31), QLTG_ERR_UNSUPPORTED, "permutation too large");
  // the block of every item goes behind the descriptors: one allocation, one copy
  host.resize(nblocks + (ntiles * sizeof(int32_t) + sizeof(PermDesc) - 1) / sizeof(PermDesc));
  int32_t* item = reinterpret_cast<int32_t*>(host.data() + nblocks);
  for (int64_t b = 0; b < nblocks; ++b)
    std::fill(item + host[b].tile_begin, item + (b + 1 < nblocks ? host[b + 1].tile_begin : ntiles), (int32_t)b);
  dev = upload(host, s);
}

void TransposeList::launch(const void* src, void* dst, int elem_bytes, cudaStream_t s) const {
  if (ntiles == 0) return;
  const PermDesc* descs = dev.as<PermDesc>();
  const int32_t* item = reinterpret_cast<const int32_t*>(descs + nblocks);
  if (elem_bytes == 8) launch_permute<double>(descs, nblocks, item, ntiles, src, dst, s);
  else launch_permute<double2>(descs, nblocks, item, ntiles, src, dst, s);
}

// ---------------------------------------------------------------------------
// Allocation-free variant (qltg_transpose_noalloc). Some callers cannot allocate device
// memory while they run - a DMRG sweep whose device memory was handed up front to another
// framework's pool (a cudaMalloc then fails or evicts that pool's cache), or a loop that
// cannot pay for the device-wide synchronisation of cudaMalloc / cudaFree - so the per-call
// permutation work list lives in this fixed device table instead of a fresh cudaMalloc.
// Every GPU that loads the library holds the table (about 850 KB) until the process exits.
// All calls share it and it keeps the last call's descriptors, so calls that overlap on the
// GPU (on different streams at once) race; each call waits for its own kernel before
// returning. The table's device address is looked up once per device and kept for the life
// of the process: the library must not outlive a cudaDeviceReset.
namespace {

__device__ __align__(256) PermDesc g_noalloc_perm[kNoAllocPermBlocks];

// Device address of the table on the current device, looked up on every call (host code
// may not use the symbol itself as a device pointer; the lookup allocates nothing, and not
// caching it keeps the address right after a device reset or a reload of the module).
PermDesc* noalloc_table(int device) {
  int cur = -1;
  QLTG_CUDA(cudaGetDevice(&cur));
  QLTG_CHECK(cur == device, QLTG_ERR_INVALID, "the no-allocation permute runs on the current device");
  void* p = nullptr;
  QLTG_CUDA(cudaGetSymbolAddress(&p, g_noalloc_perm));
  return static_cast<PermDesc*>(p);
}

}  // namespace

void launch_permute_noalloc(int device, const TransposeList& tl, const void* src, void* dst, int elem_bytes,
                            cudaStream_t s) {
  QLTG_CHECK(tl.nblocks <= kNoAllocPermBlocks, QLTG_ERR_INVALID,
             "qltg_transpose_noalloc: tensor has " + std::to_string(tl.nblocks) + " blocks, the fixed table holds " +
                 std::to_string(kNoAllocPermBlocks));
  PermDesc* table = noalloc_table(device);
  if (tl.ntiles == 0) return;
  QLTG_CUDA(cudaMemcpyAsync(table, tl.host.data(), tl.host.size() * sizeof(PermDesc), cudaMemcpyHostToDevice, s));
  if (elem_bytes == 8) launch_permute<double>(table, tl.nblocks, nullptr, tl.ntiles, src, dst, s);
  else launch_permute<double2>(table, tl.nblocks, nullptr, tl.ntiles, src, dst, s);
  // the descriptors were copied from this call's host memory and the table is shared:
  // finish before returning
  QLTG_CUDA(cudaStreamSynchronize(s));
}

}  // namespace qltg
