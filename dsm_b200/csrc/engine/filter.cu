// Cluster-encoding candidate filter on the GPU (filter.cu of the reference:
// oneRoundFilterBidirectionKernel 394-613, encode/merge/combine 615-1177,
// compact 1692-1749), run per query on the batch's union graph.
//
// The graph's runs are label-major (entries carry the label slot above the
// id).  Layout per query: vcand[v] (bit u: v passes LDF+NLF for u, the
// reference's d_v_candidate_us_), valid[v] (bit u: v is still a candidate
// of u; merges and combines clear bits, as the reference overwrites entries
// of its per-u candidate lists), enc[v * words + pos / 32] (cluster
// encodings), bitmap[u * col_len + v / 32] (per-u result, the reference's
// compact layout).  Ops run in the host plan's order, one launch each; inside
// an op the bits read belong to older clusters and the bits written to the
// op's own cluster, and every write is an atomic OR / AND, so the result does
// not depend on thread order (the reference's plain read-modify-writes next
// to atomicOr, filter.cu:688/763/868/874, can lose bits; this is their
// race-free intent).
//
// Incremental runs.  The reference recomputes the whole filter every batch
// (main.cu:213).  Here a query's state stays resident between batches, and a
// batch recomputes only the vertices whose state can differ from the previous
// batch's: the union graphs of two batches differ only in edges at endpoints
// of the two batches' updates (T), LDF+NLF of a vertex depends on its own
// adjacency, and each op moves information one hop (a core candidate's
// validity to its neighbours' leaf bits), so after D ops only vertices within
// D hops of T can differ.  For those (the region) every op is recomputed in
// pull form: a receiver takes an op's leaf bits if some neighbour is a valid
// core candidate at the op's start.  A neighbour inside the region has that
// validity in `valid` as the run proceeds; one outside kept its whole history,
// so its validity at op k is replayed from its final bits (its LDF+NLF bit and
// the checks of the merges and combines before k with the same core, which
// read bits of earlier layers that nothing rewrites later).  A region that
// outgrows its list, a state not computed in the previous batch, or a graph
// changed outside a filtered batch make the run recompute every vertex.
#include <algorithm>

#include "filter.cuh"

namespace dsm {

namespace {

__device__ __forceinline__ bool ebit(const uint32_t *enc, uint32_t words, uint32_t v, uint32_t pos) {
  return (enc[(size_t)v * words + (pos >> 5)] >> (pos & 31)) & 1u;
}
// Inside an op a bit only ever goes one way, so one that is there already (a
// hub hears from thousands of candidates) needs no atomic.
__device__ __forceinline__ void eset(uint32_t *enc, uint32_t words, uint32_t v, uint32_t pos) {
  if (!ebit(enc, words, v, pos)) atomicOr(&enc[(size_t)v * words + (pos >> 5)], 1u << (pos & 31));
}
__device__ __forceinline__ void eclr(uint32_t *enc, uint32_t words, uint32_t v, uint32_t pos) {
  if (ebit(enc, words, v, pos)) atomicAnd(&enc[(size_t)v * words + (pos >> 5)], ~(1u << (pos & 31)));
}

// Whether this run of the query recomputes every vertex.
__device__ __forceinline__ bool decide_full(const QFilterDesc *D, const RegionDevice &rg, int force_full) {
  if (force_full || rg.info == nullptr) return true;
  const RegionInfo &I = *rg.info;
  if (I.stale_now || I.prev_ov || D->hops > I.hops || I.ov_round <= D->hops) return true;
  return D->fepoch + 1 != I.epoch;  // not computed in the previous filtered batch
}

// The vertices of this run: all of them, or the query's region.
struct Scope {
  bool full;
  uint32_t count;
  const uint32_t *list;
};
__device__ __forceinline__ Scope scope_of(const QFilterDesc *D, const RegionDevice &rg, uint32_t nv) {
  Scope s;
  s.full = D->full_now != 0;
  s.list = rg.list;
  s.count = s.full ? nv : rg.info->bound[D->hops];
  return s;
}

__device__ __forceinline__ bool in_region(const RegionDevice &rg, uint32_t epoch, uint32_t hops, uint32_t v) {
  const uint32_t m = rg.mark[v];
  return (m >> 6) == epoch && (m & 63) <= hops;
}

// LDF + NLF (filter.cu:394-613): label equal, degree >= the query vertex's
// degree in the full query, and for every label l below the query's largest
// label + 1 at least as many neighbours of label l as the query vertex has.
// Clears the vertex's encodings.  The first kernel of a run: decides whether
// the run is full.
//
// Bound by the slot offsets' bytes.  A label-major run already holds a
// vertex's neighbours counted by label: lane l of the warp takes the
// difference of two slot offsets (one coalesced row of at most 132 bytes)
// where the run itself was read and every neighbour's label gathered before.
// Only slot 31, which labels above 31 share, is read when the query uses label
// 31.  A warp takes 32 vertices, so that labels, degrees and results move as
// 128-byte rows and vertices without a query label cost nothing more.
// 2^20 vertices, 2^24 edges, one query: 325 -> 41 us.
__global__ void k_ldf_nlf(DevGraph g, const FilterDevice *F, RegionDevice rg, int force_full) {
  const FilterDevice f = F[blockIdx.y];
  QFilterDesc *D = f.desc;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  const uint32_t nl = D->nlabels, words = f.words;
  const bool full = decide_full(D, rg, force_full);
  if (blockIdx.x == 0 && threadIdx.x == 0) D->full_now = full ? 1u : 0u;
  const uint32_t count = full ? g.nv : rg.info->bound[D->hops];
  for (uint32_t base = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32; base < count; base += warps * 32) {
    const uint32_t i = base + lane;
    const uint32_t v = i < count ? (full ? i : rg.list[i]) : 0u;
    uint32_t keep = 0, res = 0;
    if (i < count) {
      const uint32_t lv = g.lab[v] & kLabelMask, dv = g.adj[v].y;
      for (uint32_t b = lv < nl ? D->label_us[lv] : 0u; b; b &= b - 1) {  // query vertices with this label
        const uint32_t u = __ffs(b) - 1;
        if (D->qdeg[u] <= dv) keep |= 1u << u;
      }
    }
    for (uint32_t m = __ballot_sync(kFull, keep != 0); m; m &= m - 1) {
      const uint32_t k = __ffs(m) - 1;
      const uint32_t vk = __shfl_sync(kFull, v, k), kk = __shfl_sync(kFull, keep, k);
      const uint32_t *t = g.loff + (size_t)vk * (g.nlt + 1);
      const uint32_t a = lane <= g.nlt ? t[lane] : 0u;
      uint32_t b = __shfl_down_sync(kFull, a, 1);
      if (lane == 31 && g.nlt == 32) b = t[32];
      uint32_t mine = lane < g.nlt ? b - a : 0u;
      if (nl == 32 && g.nlt == 32) {  // slot 31 holds every label >= 31: count label 31 itself
        const uint32_t lo = __shfl_sync(kFull, a, 31), hi = __shfl_sync(kFull, b, 31);
        const uint32_t *run = adj_list(g, g.adj[vk]);
        uint32_t c = 0;
        for (uint32_t j = lo + lane; j < hi; j += 32) c += (g.lab[run[j] & kIdMask] & kLabelMask) == 31;
        c = __reduce_add_sync(kFull, c);
        if (lane == 31) mine = c;
      }
      uint32_t rk = 0;
      for (uint32_t b2 = kk; b2; b2 &= b2 - 1) {
        const uint32_t u = __ffs(b2) - 1;
        if (__all_sync(kFull, lane >= nl || mine >= D->nlc[u][lane])) rk |= 1u << u;
      }
      if (lane == k) res = rk;
    }
    if (i < count) {
      f.vcand[v] = res;
      f.valid[v] = res;
    }
    if (full) {
      const size_t e0 = (size_t)base * words, e1 = (size_t)min(base + 32, count) * words;
      for (size_t e = e0 + lane; e < e1; e += 32) f.enc[e] = 0;
    } else if (i < count) {
      for (uint32_t w = 0; w < words; ++w) f.enc[(size_t)v * words + w] = 0;
    }
  }
}

// The core rule of op k for candidate c (valid for the op's core at its start).
__device__ __forceinline__ void core_rule(const DevFilterOp &op, uint32_t c, uint32_t *valid, uint32_t *enc,
                                          uint32_t words) {
  const uint32_t cu = op.core_u, pos = op.pos;
  if (op.kind == 0) {  // encodeKernel: core bit
    eset(enc, words, c, pos);
  } else if (op.kind == 1) {  // mergeKernel: both parents' bits of the core
    if (ebit(enc, words, c, op.lp) && ebit(enc, words, c, op.rp)) eset(enc, words, c, pos);
    else atomicAnd(&valid[c], ~(1u << cu));
  } else {  // combineMultipleClustersKernel: every small cluster's core bit
    bool all = true;
    for (uint32_t s = 0; s < op.nsmall; ++s) all = all && ebit(enc, words, c, op.small_core_pos[s]);
    if (all) {
      if (op.comb_type == 0) eset(enc, words, c, pos);
    } else {
      eclr(enc, words, c, pos);
      atomicAnd(&valid[c], ~(1u << cu));
    }
  }
}

// The leaf rule of op k for receiver n (a neighbour of a valid core candidate).
__device__ __forceinline__ void leaf_rule(const DevFilterOp &op, uint32_t n, const uint32_t *vcand, uint32_t *enc,
                                          uint32_t words) {
  const uint32_t pos = op.pos;
  if (op.kind == 0) {
    const uint32_t code = vcand[n];
    for (uint32_t j = 0; j < op.nleaf; ++j)
      if ((code >> op.leaf_u[j]) & 1u) eset(enc, words, n, pos + 1 + j);
  } else if (op.kind == 1) {
    if (ebit(enc, words, n, op.lcp)) eset(enc, words, n, pos + 1);
    if (op.rcp != op.rp && ebit(enc, words, n, op.rcp)) eset(enc, words, n, pos + 2);
  } else {
    for (uint32_t j = 0; j < op.nleaf; ++j) {
      bool fv = true;
      for (uint32_t t = 0; t < op.leaf_src_count[j]; ++t) fv = fv && ebit(enc, words, n, op.leaf_src[j][t]);
      if (op.comb_type == 1) {
        if (!fv) eclr(enc, words, n, pos + 1 + j);
      } else if (fv) {
        eset(enc, words, n, pos + 1 + j);
      }
    }
  }
}

// The ranges of a block's 256 vertices (thread t: len entries from arena word
// `first`) laid end to end: incl is the inclusive scan of the lengths, entry
// e of the total lies at arena word start[o] + e for its owner o.  Longer ranges
// are laid in rounds of kSpan entries a vertex, so that 256 of them count in 32
// bits (a vertex has up to 2^27 neighbours).
#ifndef DSM_RANGE_SPAN  // tests build with a small one
#define DSM_RANGE_SPAN (1u << 23)
#endif
constexpr uint32_t kSpan = DSM_RANGE_SPAN;
struct BlockRanges {
  unsigned long long start[256];
  uint32_t incl[256];
  uint32_t warp[8];
};
__device__ __forceinline__ uint32_t lay_ranges(BlockRanges &R, unsigned long long first, uint32_t len) {
  const uint32_t t = threadIdx.x, lane = t & 31;
  uint32_t incl = len;
#pragma unroll
  for (uint32_t d = 1; d < 32; d <<= 1) {
    const uint32_t x = __shfl_up_sync(kFull, incl, d);
    if (lane >= d) incl += x;
  }
  if (lane == 31) R.warp[t >> 5] = incl;
  __syncthreads();
  for (uint32_t w = 0; w < (t >> 5); ++w) incl += R.warp[w];
  R.incl[t] = incl;
  R.start[t] = first - (incl - len);
  __syncthreads();
  return R.incl[255];
}
__device__ __forceinline__ unsigned long long range_entry(const BlockRanges &R, uint32_t e) {
  uint32_t o = 0;  // the first owner with incl > e
#pragma unroll
  for (uint32_t d = 128; d; d >>= 1)
    if (R.incl[o + d - 1] <= e) o += d;
  return R.start[o] + e;
}

// Full runs: one op over every current candidate of its core vertex.
//
// Bound by the latency of the steps (candidates, offsets, scan, entries,
// receivers): few vertices are candidates.  Only neighbours of the labels the
// leaf rule can change are visited (leaf_slots: one contiguous range each of
// the label-major run).  A block looks through 1024 vertices at a time and
// gathers the candidates; 256 of them, or the last, a thread each, have their
// ranges of one label laid end to end (a block scan of their lengths), and each
// thread takes one entry in turn, its owner found by eight steps through the
// scan: a hub's range is then shared by the block, where one warp walked the
// hub's whole run before and the launch waited for it.  2^20 vertices, 2^24
// edges (R-MAT), one op: 635 us; 46 us with the ranges of every 256 vertices
// laid out, most of them no candidates; 33 us so.
constexpr uint32_t kOpTile = 1024;
__global__ void __launch_bounds__(256) k_filter_op(DevGraph g, const FilterDevice *F, uint32_t k) {
  const FilterDevice f = F[blockIdx.y];
  if (k >= f.nops || !f.desc->full_now) return;
  __shared__ BlockRanges R;
  __shared__ uint32_t s_cand[256 + kOpTile];
  // candidates gathered, of even and odd tiles: what a tile leaves goes to the
  // other one's, so that no thread still reads what is written
  __shared__ uint32_t s_n[2];
  const DevFilterOp &op = f.ops[k];
  const uint32_t t = threadIdx.x, lane = t & 31, cu = op.core_u, words = f.words;
  if (t < 2) s_n[t] = 0;
  __syncthreads();
  uint32_t odd = 0;
  for (uint32_t base = blockIdx.x * kOpTile; base < g.nv; base += gridDim.x * kOpTile, odd ^= 1) {
    const bool last = base + gridDim.x * kOpTile >= g.nv || base + gridDim.x * kOpTile < base;
#pragma unroll
    for (uint32_t i = 0; i < kOpTile; i += 256) {
      const uint32_t v = base + i + t;
      const bool isc = v < g.nv && ((f.valid[v] >> cu) & 1u);
      const uint32_t m = __ballot_sync(kFull, isc);
      uint32_t at = 0;
      if (m && lane == 0) at = atomicAdd(&s_n[odd], (uint32_t)__popc(m));
      at = __shfl_sync(kFull, at, 0);
      if (isc) s_cand[at + __popc(m & lanemask_lt())] = v;
    }
    __syncthreads();
    uint32_t n = s_n[odd];
    while (n >= 256 || (last && n)) {
      const uint32_t take = min(n, 256u);
      n -= take;
      const bool isc = t < take;
      const uint32_t v = isc ? s_cand[n + t] : 0u;
      uint32_t off = 0;
      if (isc) {
        core_rule(op, v, f.valid, f.enc, words);
        off = g.adj[v].x;
      }
      for (uint32_t sm = op.leaf_slots; sm; sm &= sm - 1) {
        const uint32_t sl = __ffs(sm) - 1;
        if (sl >= g.nlt) break;  // no vertex has a label of this slot or a later one
        uint32_t a = 0, len = 0;
        if (isc) {
          const uint32_t *lo = g.loff + (size_t)v * (g.nlt + 1) + sl;
          a = lo[0];
          len = lo[1] - a;
        }
        uint32_t total;
        do {
          total = lay_ranges(R, (unsigned long long)off * 4 + a, min(len, kSpan));
          for (uint32_t e = t; e < total; e += 256)
            leaf_rule(op, g.arena[range_entry(R, e)] & kIdMask, f.vcand, f.enc, words);
          __syncthreads();
          a += kSpan;
          len -= min(len, kSpan);
        } while (total >= kSpan);  // below it no vertex has more
      }
    }
    if (t == 0) s_n[odd ^ 1] = n;
    __syncthreads();
  }
}

// Validity of c for the core of op k at the op's start, for a vertex outside
// the region (its bits are those of the previous run, which it shares).
__device__ __forceinline__ bool replayed_valid(const DevFilterOp *ops, const DevFilterOp &op, uint32_t c,
                                               const uint32_t *vcand, const uint32_t *enc, uint32_t words) {
  if (!((vcand[c] >> op.core_u) & 1u)) return false;
  for (uint32_t p = 0; p < op.nprior; ++p) {
    const DevFilterOp &q = ops[op.prior[p]];
    if (q.kind == 1) {
      if (!(ebit(enc, words, c, q.lp) && ebit(enc, words, c, q.rp))) return false;
    } else {
      for (uint32_t s = 0; s < q.nsmall; ++s)
        if (!ebit(enc, words, c, q.small_core_pos[s])) return false;
    }
  }
  return true;
}

// Region runs, op k, first half: every receiver of the region pulls its
// leaf bits (a warp per receiver scans its neighbours of the core's label for
// a valid core candidate at the op's start).
__global__ void k_filter_pull(DevGraph g, const FilterDevice *F, uint32_t k, RegionDevice rg) {
  const FilterDevice f = F[blockIdx.y];
  const QFilterDesc *D = f.desc;
  if (k >= f.nops || D->full_now) return;
  const DevFilterOp &op = f.ops[k];
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  const uint32_t epoch = rg.info->epoch, hops = D->hops, words = f.words;
  const uint32_t count = rg.info->bound[hops];
  const uint32_t cu = op.core_u, sl = op.core_slot;
  if (sl >= g.nlt) return;  // no candidates
  for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < count; i += warps) {
    const uint32_t n = rg.list[i];
    const uint32_t *run = adj_list(g, g.adj[n]);
    const uint32_t *lo = g.loff + (size_t)n * (g.nlt + 1) + sl;
    const uint32_t end = lo[1];
    bool has = false;
    for (uint32_t b = lo[0]; b < end && !has; b += 32) {
      bool cv = false;
      if (b + lane < end) {
        const uint32_t c = run[b + lane] & kIdMask;
        cv = in_region(rg, epoch, hops, c) ? ((f.valid[c] >> cu) & 1u) != 0
                                           : replayed_valid(f.ops, op, c, f.vcand, f.enc, words);
      }
      has = __any_sync(kFull, cv);
    }
    if (has && lane == 0) leaf_rule(op, n, f.vcand, f.enc, words);
  }
}

// Region runs, op k, second half: the core rule for the region's candidates.
__global__ void k_filter_core(const FilterDevice *F, uint32_t k, RegionDevice rg) {
  const FilterDevice f = F[blockIdx.y];
  const QFilterDesc *D = f.desc;
  if (k >= f.nops || D->full_now) return;
  const DevFilterOp &op = f.ops[k];
  const uint32_t count = rg.info->bound[D->hops];
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
    const uint32_t c = rg.list[i];
    if ((f.valid[c] >> op.core_u) & 1u) core_rule(op, c, f.valid, f.enc, f.words);
  }
}

// compact (filter.cu:1692-1749): bitmap[u][v / 32] from the bit at u's
// position (or, with LDF+NLF only, from vcand).  Full runs: a warp per word;
// region runs: a warp per region vertex, rewriting its whole word.  The
// last kernel of a run: records the epoch the state belongs to.
__global__ void k_filter_compact(uint32_t nv, const FilterDevice *F, int ldf_only, RegionDevice rg) {
  const FilterDevice f = F[blockIdx.y];
  QFilterDesc *D = f.desc;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  const Scope sc = scope_of(D, rg, nv);
  const uint32_t count = sc.full ? f.col_len : sc.count;
  for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < count; i += warps) {
    const uint32_t w = sc.full ? i : (sc.list[i] >> 5);
    const uint32_t v = w * 32 + lane;
    for (uint32_t u = 0; u < D->nq; ++u) {
      bool b = false;
      if (v < nv) b = ldf_only ? ((f.vcand[v] >> u) & 1u) : ebit(f.enc, f.words, v, D->pos_of_u[u]);
      uint32_t m = __ballot_sync(kFull, b);
      if (lane == 0) f.bitmap[(size_t)u * f.col_len + w] = m;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) D->fepoch = rg.info ? rg.info->epoch : 0xFFFFFFFFu;
}

// ---- region ----------------------------------------------------------------
__device__ __forceinline__ void claim(const RegionDevice &rg, uint32_t epoch, uint32_t v, uint32_t hop) {
  const uint32_t old = rg.mark[v];
  if ((old >> 6) == epoch) return;
  if (atomicCAS(&rg.mark[v], old, (epoch << 6) | hop) != old) return;  // claimed by another thread
  const uint32_t idx = atomicAdd(&rg.info->total, 1u);
  if (idx < rg.info->cap) rg.list[idx] = v;
  else atomicMin(&rg.info->ov_round, hop);
}

__global__ void k_region_begin(RegionInfo *I, uint32_t hops) {
  I->stale_now = I->stale;
  I->stale = 0;
  I->epoch = (I->epoch + 1) & 0x03FFFFFFu;
  if (I->epoch == 0) I->epoch = 1;
  I->total = 0;
  I->ov_round = 64;
  I->hops = hops;
}

__global__ void k_region_seed(DevGraph g, RegionDevice rg, const uint32_t *hdr_n, const uint4 *upd) {
  const uint32_t n = *hdr_n, epoch = rg.info->epoch, np = rg.info->prev_cnt;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < 2 * n + np; i += gridDim.x * blockDim.x) {
    uint32_t v;
    if (i < 2 * n) {
      const uint4 u = upd[i >> 1];
      v = (i & 1) ? u.z : u.y;
    } else {
      v = rg.prev[i - 2 * n];
    }
    if (v < g.nv) claim(rg, epoch, v, 0);
  }
}

__global__ void k_region_close(RegionInfo *I, uint32_t hop) { I->bound[hop] = min(I->total, I->cap); }

// Hop `hop`: every neighbour of the vertices first reached at hop - 1.  A
// block shares the runs of up to 256 of them, fewer while there are blocks
// without any (a warp per run left the launch waiting for the warps that had
// drawn the hubs, and one block for the first hop's 256 vertices for that block).
__global__ void __launch_bounds__(256) k_region_expand(DevGraph g, RegionDevice rg, uint32_t hop) {
  __shared__ BlockRanges R;
  const RegionInfo &I = *rg.info;
  // The list is full: queries that far out run in full.  Other blocks of this
  // launch may lower the word meanwhile, so the block decides as one.
  if (__syncthreads_or(*(volatile const uint32_t *)&rg.info->ov_round < 64)) return;
  const uint32_t lo = hop >= 2 ? I.bound[hop - 2] : 0u, hi = I.bound[hop - 1];
  const uint32_t t = threadIdx.x, epoch = I.epoch;
  const uint32_t tile = min((hi - lo + gridDim.x - 1) / gridDim.x, 256u);
  for (uint32_t base = lo + blockIdx.x * tile; base < hi; base += gridDim.x * tile) {
    const uint2 av = t < tile && base + t < hi ? g.adj[rg.list[base + t]] : make_uint2(0, 0);
    unsigned long long first = (unsigned long long)av.x * 4;
    uint32_t len = av.y, total;
    do {
      total = lay_ranges(R, first, min(len, kSpan));
      for (uint32_t e = t; e < total; e += 256) {
        claim(rg, epoch, g.arena[range_entry(R, e)] & kIdMask, hop);
        if ((e >> 8) % 8 == 7 && *(volatile const uint32_t *)&rg.info->ov_round < 64) break;
      }
      if (__syncthreads_or(*(volatile const uint32_t *)&rg.info->ov_round < 64)) return;
      first += kSpan;
      len -= min(len, kSpan);
    } while (total >= kSpan);  // below it no vertex has more
  }
}

// The batch's endpoints become the next batch's previous endpoints.
__global__ void k_region_save(RegionDevice rg, const uint32_t *hdr_n, const uint4 *upd) {
  const uint32_t n = *hdr_n, cap = rg.info->prev_cap;
  const bool fits = 2ull * n <= cap;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n && fits; i += gridDim.x * blockDim.x) {
    const uint4 u = upd[i];
    rg.prev[2 * i] = u.y;
    rg.prev[2 * i + 1] = u.z;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    rg.info->prev_cnt = fits ? 2 * n : 0u;
    rg.info->prev_ov = fits ? 0u : 1u;
  }
}

}  // namespace

int launch_query_filters(const DevGraph &g, const FilterDevice *f, uint32_t nf, uint32_t max_ops, int mode,
                         int num_sms, cudaStream_t s, const RegionDevice &rg, int force_full) {
  if (nf == 0) return 0;
  // queries share the launch: about 16 blocks per SM over all of them, and
  // never fewer than an SM's worth of one query's
  const unsigned per = std::max<unsigned>(num_sms * 16u / nf, num_sms);
  int launched = 0;
  for (uint32_t q0 = 0; q0 < nf; q0 += 65535u) {  // the grid's limit in y
    const uint32_t nq = std::min(nf - q0, 65535u);
    const FilterDevice *fq = f + q0;
    const dim3 grid(per, nq), light(std::min<unsigned>(per, num_sms * 2u), nq);
    k_ldf_nlf<<<grid, 256, 0, s>>>(g, fq, rg, force_full);
    ++launched;
    for (uint32_t k = 0; mode >= 2 && k < max_ops; ++k) {
      k_filter_op<<<grid, 256, 0, s>>>(g, fq, k);
      ++launched;
      if (rg.info && !force_full) {
        k_filter_pull<<<grid, 256, 0, s>>>(g, fq, k, rg);
        k_filter_core<<<light, 256, 0, s>>>(fq, k, rg);
        launched += 2;
      }
    }
    k_filter_compact<<<grid, 256, 0, s>>>(g.nv, fq, mode < 2, rg);
    ++launched;
  }
  return launched;
}

void launch_region_build(const DevGraph &g, const RegionDevice &rg, const uint32_t *hdr_n, const uint4 *upd,
                         uint32_t hops, int num_sms, cudaStream_t s) {
  k_region_begin<<<1, 1, 0, s>>>(rg.info, hops);
  k_region_seed<<<num_sms * 4, 256, 0, s>>>(g, rg, hdr_n, upd);
  k_region_close<<<1, 1, 0, s>>>(rg.info, 0);
  for (uint32_t h = 1; h <= hops; ++h) {
    k_region_expand<<<num_sms * 8, 256, 0, s>>>(g, rg, h);
    k_region_close<<<1, 1, 0, s>>>(rg.info, h);
  }
}

void launch_region_save(const RegionDevice &rg, const uint32_t *hdr_n, const uint4 *upd, cudaStream_t s) {
  k_region_save<<<64, 256, 0, s>>>(rg, hdr_n, upd);
}

}  // namespace dsm
