// Contraction execution: schedule construction after device pairing, and the launch
// sequence (operand transposes, then one grouped GEMM).
#include <algorithm>
#include <cstring>

#include "ctrct.h"
#include "split.h"

namespace qltg {

// FP64 warp tiles (bm / 4 rows x kF64TileCols columns, gemm_f64.cu), longest first. All tiles of
// a block with the same extent inside it cost the same, so the list holds at most four runs per
// block instead of every tile.
static void f64_tile_list(GemmSchedule& g, int num_sms) {
  g.run.clear();
  g.ntiles = 0;
  struct Cand { GemmTileRun r; int64_t count, cost; };
  std::vector<Cand> cands;
  const int rows = g.bm / 4, cols = kF64TileCols;
  // multiply-adds issued for an extent: whole 8 x 4 pieces
  auto padded = [](int64_t r, int64_t c) { return ((r + 7) / 8 * 8) * ((c + 3) / 4 * 4); };
  for (int32_t q = 0; q < (int32_t)g.cblk.size(); ++q) {
    const GemmCBlk& cb = g.cblk[q];
    if (skinny_cblk(g, q)) continue;
    QLTG_CHECK((cb.m + 31) / 32 < 32768 && (cb.n + 31) / 32 < 32768, QLTG_ERR_UNSUPPORTED,
               "output block too large for the tile grid");
    int64_t ksum = 0;
    for (int32_t t = cb.t0; t < cb.t1; ++t) ksum += g.task[t].k;
    const int fm = cb.m / rows, fn = cb.n / cols, em = cb.m % rows, en = cb.n % cols;
    auto add = [&](int tm0, int tn0, int nm, int nn, int r, int c) {
      if (nm > 0 && nn > 0) cands.push_back({GemmTileRun{q, 0, tm0, tn0, nn}, (int64_t)nm * nn, ksum * padded(r, c)});
    };
    add(0, 0, fm, fn, rows, cols);
    add(0, fn, fm, en ? 1 : 0, rows, en);
    add(fm, 0, em ? 1 : 0, fn, em, cols);
    add(fm, fn, em ? 1 : 0, en ? 1 : 0, em, en);
  }
  std::stable_sort(cands.begin(), cands.end(), [](const Cand& x, const Cand& y) { return x.cost > y.cost; });
  // Tiles are shared by a CTA's four warps when the longest one, alone on its sub-partition,
  // would take more than a quarter of a sub-partition's share of the launch (four per SM): with
  // four warps resident on each, one such tile then ends the launch late. All or none: sharing
  // only the longest ones left the rest to start late (FP64 step 3 of the matvec: D = 1000 280 us
  // own / 266 us shared / 362-449 us mixed, D = 300 82 / 51 us; steps above the line, D = 4000:
  // 2.52-2.58 ms own, 2.75-2.78 ms shared).
  double total = 0;
  for (auto& c : cands) total += (double)c.cost * c.count;
  g.share_tiles = !cands.empty() && 4.0 * cands[0].cost > total / (4.0 * std::max(1, num_sms));
  g.run.reserve(cands.size());
  for (auto& c : cands) {
    QLTG_CHECK(g.ntiles + c.count < ((int64_t)1 << 31) - (1 << 20), QLTG_ERR_UNSUPPORTED, "too many output tiles");
    c.r.begin = (int32_t)g.ntiles;
    g.ntiles += c.count;
    g.run.push_back(c.r);
  }
}

void set_f64_tile(CtrctPlan& p, int bm, cudaStream_t s) {
  QLTG_CHECK(bm == 32 || bm == 64, QLTG_ERR_INVALID, "FP64 tiles have 32 or 64 rows");
  GemmSchedule& g = p.sched;
  if (g.bm == bm && g.d_run.get()) return;
  g.bm = bm;
  f64_tile_list(g, p.ctx->num_sms);
  g.d_run = upload(g.run, s);
  QLTG_CUDA(cudaStreamSynchronize(s));
}

// Entries and pieces of the skinny blocks (the tasks' operand offsets are final). An item is one
// pass of a warp, 128 outputs; where there are very many passes and blocks are large enough for it
// to add under a quarter of empty ones, an item stands for four passes, to keep the list short.
static void skinny_list(GemmSchedule& g, int num_sms) {
  int64_t passes = 0, items = 0;
  g.skinny_long = false;
  for (int32_t q = 0; q < (int32_t)g.cblk.size(); ++q) {
    if (!skinny_cblk(g, q)) continue;
    const int64_t outputs = (int64_t)g.cblk[q].m * g.cblk[q].n;
    g.skinny_long |= outputs >= ((int64_t)1 << 31) - 512;   // (a pass counts on past the block's end)
    passes += (outputs + 127) / 128;
    items += (outputs + 511) / 512;
  }
  g.skinny_outputs = passes > (int64_t)num_sms * 32 * 4 && 16 * items <= 5 * passes ? 512 : 128;
  QLTG_CHECK(4 * items < ((int64_t)1 << 31) && passes < ((int64_t)1 << 31), QLTG_ERR_UNSUPPORTED, "too many rows of small blocks");
  for (int32_t q = 0; q < (int32_t)g.cblk.size(); ++q) {
    if (!skinny_cblk(g, q)) continue;
    const GemmCBlk& cb = g.cblk[q];
    const size_t e0 = g.skinny_entry.size();
    for (int32_t t = cb.t0; t < cb.t1; ++t) {
      const GemmTask& tk = g.task[t];
      for (int32_t kk = 0; kk < tk.k; ++kk)
        g.skinny_entry.push_back(SkinnyEntry{tk.a_off + (int64_t)kk * tk.a_cs, tk.b_off + (int64_t)kk * cb.n, tk.a_rs, tk.sign, 0});
    }
    QLTG_CHECK(g.skinny_entry.size() < ((size_t)1 << 31), QLTG_ERR_UNSUPPORTED, "too many small tasks");
    for (int64_t o = 0; o < (int64_t)cb.m * cb.n; o += g.skinny_outputs)
      g.skinny.push_back(SkinnyItem{q, (int32_t)(o / 128), (int32_t)e0, (int32_t)g.skinny_entry.size()});
  }
}

void finalize_plan(CtrctPlan& p, cudaStream_t s) {
  GemmSchedule& g = p.sched;
  g.skinny.clear();
  g.skinny_entry.clear();
  bool any_skinny = false;
  for (int32_t q = 0; q < (int32_t)g.cblk.size(); ++q) any_skinny |= skinny_cblk(g, q);
  f64_tile_list(g, p.ctx->num_sms);
  // Operand transposes. A task reads its operand block from the transposed scratch unless
  // (a) the permutation leaves the block's layout unchanged, or (b) it is a skinny task and
  // the block, read in place, is a strided matrix (rows and columns each one stride); such
  // tasks read the operand itself (offset flag kFromSrc) and blocks nobody reads from the
  // scratch get no transpose work.
  const size_t eb = p.a.elem_bytes();
  const bool any_work = g.ntiles || any_skinny;
  std::vector<uint8_t> skinny_task(g.task.size(), 0);
  for (int32_t q = 0; q < (int32_t)g.cblk.size(); ++q)
    if (skinny_cblk(g, q))
      for (int32_t t = g.cblk[q].t0; t < g.cblk[q].t1; ++t) skinny_task[t] = 1;
  auto block_of = [](const Meta& m, int64_t off) {
    const int64_t b = std::lower_bound(m.offsets.begin(), m.offsets.end(), off) - m.offsets.begin();
    QLTG_CHECK(b < m.nblk && m.offsets[b] == off, QLTG_ERR_INVALID, "internal: task operand offset is no block start");
    return b;
  };
  // (row stride, column stride) of block b of A read in place, rows = saved legs, columns =
  // contracted legs in the transposed order; false if either needs more than one stride
  auto strided_a = [&](int64_t b, int32_t& rs, int32_t& cs) {
    const int r = p.a.rank, ns = (int)p.sa.size();
    std::vector<int64_t> sstr(r);
    if (r) sstr[r - 1] = 1;
    for (int i = r - 2; i >= 0; --i) sstr[i] = sstr[i + 1] * p.a.dim(b, i + 1);
    auto merge = [&](int lo, int hi, int32_t& stride) {
      int64_t run_dim = 0, run_stride = 1;
      int n = 0;
      for (int i = lo; i < hi; ++i) {
        const int leg = p.a_order[i];
        const int64_t d = p.a.dim(b, leg);
        if (d == 1) continue;
        if (n && run_stride == sstr[leg] * d) {
          run_dim *= d;
          run_stride = sstr[leg];
        } else {
          if (n) return false;
          run_dim = d;
          run_stride = sstr[leg];
          n = 1;
        }
      }
      if (run_stride >= ((int64_t)1 << 31)) return false;
      stride = (int32_t)(n ? run_stride : 0);
      return true;
    };
    return merge(0, ns, rs) && merge(ns, r, cs);
  };
  p.a_tl = TransposeList();
  p.b_tl = TransposeList();
  if (p.a_trans && p.a.size && any_work) {
    TransposeList probe;
    probe.describe(p.a, p.a_order, {}, nullptr);
    std::vector<uint8_t> need(p.a.nblk, 0);
    for (size_t t = 0; t < g.task.size(); ++t) {
      GemmTask& tk = g.task[t];
      const int64_t b = block_of(p.a, tk.a_off);
      int32_t rs = 0, cs = 0;
      if (probe.identity[b]) {
        tk.a_off |= kFromSrc;
      } else if (skinny_task[t] && strided_a(b, rs, cs)) {
        tk.a_off |= kFromSrc;
        tk.a_rs = rs;
        tk.a_cs = cs;
      } else {
        need[b] = 1;
      }
    }
    std::vector<uint8_t> skip(p.a.nblk);
    for (int64_t b = 0; b < p.a.nblk; ++b) skip[b] = !need[b];
    p.a_tl.build(p.a, p.a_order, {}, nullptr, s, false, &skip);
    if (p.a_tl.ntiles) p.a_t.alloc(p.a.size * eb);
  }
  if (p.b_trans && p.b.size && any_work) {
    p.b_tl.build(p.b, p.b_order, {}, nullptr, s, /*skip_identity=*/true);
    for (auto& tk : g.task)
      if (p.b_tl.identity[block_of(p.b, tk.b_off)]) tk.b_off |= kFromSrc;
    if (p.b_tl.ntiles) p.b_t.alloc(p.b.size * eb);
  }
  if (any_skinny) skinny_list(g, p.ctx->num_sms);
  if (any_skinny) (void)skinny_grid((int)g.skinny.size(), p.a.dtype == QLTG_C128, p.ctx->num_sms);
  // the schedule's lists in one buffer, with one copy
  {
    const struct { const void* src; size_t bytes; DevBuf* part; } lists[] = {
        {g.cblk.data(), g.cblk.size() * sizeof(GemmCBlk), &g.d_cblk},
        {g.task.data(), g.task.size() * sizeof(GemmTask), &g.d_task},
        {g.run.data(), g.run.size() * sizeof(GemmTileRun), &g.d_run},
        {g.skinny.data(), g.skinny.size() * sizeof(SkinnyItem), &g.d_skinny},
        {g.skinny_entry.data(), g.skinny_entry.size() * sizeof(SkinnyEntry), &g.d_entry},
        {nullptr, sizeof(int), &g.d_counter}};
    auto room = [](size_t n) { return (n + 255) / 256 * 256; };
    size_t total = 0;
    for (const auto& l : lists) total += room(l.bytes);
    std::vector<char> image(total, 0);
    g.lists.alloc(total);
    size_t at = 0;
    for (const auto& l : lists) {
      if (l.src) std::memcpy(image.data() + at, l.src, l.bytes);
      *l.part = DevBuf::part(g.lists, at, l.bytes);
      at += room(l.bytes);
    }
    QLTG_CUDA(cudaMemcpyAsync(g.lists.get(), image.data(), total, cudaMemcpyHostToDevice, s));
    QLTG_CUDA(cudaStreamSynchronize(s));   // before the image goes, and before any stream uses the lists
  }
  p.launches_per_exec = (g.ntiles ? 2 : 0) + (g.skinny.empty() ? 0 : 1) +   // memset + GEMM
                         (p.a_tl.ntiles ? 1 : 0) + (p.b_tl.ntiles ? 1 : 0);
}

// Kernel launches of one split-mode execution: operand transposes plus the split stage.
int64_t exec_launches_split(const CtrctPlan& p) {
  int64_t n = split_launches(p);
  if (p.a_tl.ntiles && !(p.split && p.split->a_static)) n += 1;
  if (p.b_tl.ntiles && !(p.split && p.split->b_static)) n += 1;
  return n;
}

void exec_contraction(CtrctPlan& p, const void* a, const void* b, void* c, int mode, cudaStream_t s, int stage) {
  if (!p.sched.ntiles && p.sched.skinny.empty()) return;
  QLTG_CHECK(a && b && c, QLTG_ERR_INVALID, "null device buffer");
  QLTG_CHECK(stage >= 0 && stage <= 3, QLTG_ERR_INVALID, "stage must be 0, 1, 2 or 3");
  QLTG_CHECK(mode == QLTG_MODE_FP64 || mode == QLTG_MODE_SPLIT, QLTG_ERR_INVALID, "unknown arithmetic mode");
  const int eb = (int)p.a.elem_bytes();
  // operand scratch (transposed blocks) and the operands themselves (blocks flagged
  // kFromSrc); untransposed operands are their own scratch
  Operands op{a, a, b, b};
  // operands packed once for the split path (constant for the plan's life) need no transpose
  const bool a_packed = mode == QLTG_MODE_SPLIT && p.split && p.split->a_static && p.split->a_ready;
  const bool b_packed = mode == QLTG_MODE_SPLIT && p.split && p.split->b_static && p.split->b_ready;
  if (p.a_tl.ntiles) {
    if (stage < 2 && !a_packed) p.a_tl.launch(a, p.a_t.get(), eb, s);
    op.a = p.a_t.get();
  }
  if (p.b_tl.ntiles) {
    if (stage < 2 && !b_packed) p.b_tl.launch(b, p.b_t.get(), eb, s);
    op.b = p.b_t.get();
  }
  if (stage == 1) return;
  // the FP64 kernels work on whole elements; the slices of split precision are made from FP64 values
  check_aligned(mode == QLTG_MODE_FP64 || !p.sched.skinny.empty() ? eb : sizeof(double), {a, b, c});
  if (mode == QLTG_MODE_FP64)
    launch_gemm_f64(p.sched, op, c, p.a.dtype == QLTG_C128, p.ctx->num_sms, s);
  else
    launch_gemm_split(p, op, c, s, /*pack=*/stage != 3);
}

}  // namespace qltg
