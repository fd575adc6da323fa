// Persistent DFS matcher (replaces gpu_match.cu:96-1119, join.cu:18-221 and
// the work queue of queue.cuh / job_queue.cuh).
//
// One warp per task.  A task fixes positions 0..depth-1 of a matching order
// and enumerates the rest depth-first, up to 32 partial embeddings of a level
// at a time, a lane each: their candidate ranges are laid end to end and
// scanned 32 entries a step, each lane testing one entry (injectivity, filter
// bit, membership in the other backward neighbours' label ranges, liveness at
// the update's view time), and 32 survivors make the next level's batch.
// Nothing is materialised, except, with breadth-first levels, the rows a first
// launch hands to a second.
//
// Scheduling.  Tasks are first the seeds (one atomicAdd each), then donated
// jobs.  An idle warp takes a ticket (one atomicAdd on pop_cnt) and waits for
// its own job slot to be published, polling only that slot's flag with
// exponential backoff.  Busy warps see pop_cnt - push_cnt warps waiting and
// donate to them from their shallowest level with a substantial piece: partial
// embeddings with at least two levels below them, or half of the entries left.  The warp whose task
// completion brings `outstanding` to zero sets `done` and marks every
// still-waiting ticket's slot as finished.  Every wait is bounded by a clock
// budget that restarts whenever busy warps show progress.

#include "kernels.cuh"

namespace dsm {

namespace {

template <class T>
__device__ __forceinline__ T ld_volatile(const T &x) {
  return *(const volatile T *)&x;
}

constexpr unsigned long long kSeqDone = 1ull << 63;
// Partial embeddings between heartbeats when tuples count towards a listing
// budget: those listed before a search is found over its limit count, so a
// later stop lists fewer queries, an earlier one more.  Against one partial at
// a time (a heartbeat every 64 chunks) over 156 batches, queries listed more /
// fewer: chunks alone 55 / 684, 640 252 / 442, 576 304 / 398, 400 717 / 187,
// 256 1383 / 37; two runs of one build differ by 110 / 106.  One listed request
// on 2^24 edges: 7.3 -> 6.7 ms; a count keeps 64 chunks.
constexpr uint32_t kListBeat = 576;

// Lane 0 only.  Returns 1 (seed `slot`), 2 (job of ticket `slot`; the caller
// releases the ring slot after reading it) or 0 (no more work).
__device__ uint32_t acquire(const MatchArgs &P, unsigned long long &slot, bool &seeds_done) {
  Sched *sc = P.sc;
  if (!seeds_done) {
    const unsigned long long nseeds = ld_volatile(sc->nseeds);
    if (ld_volatile(sc->seed_next.v) < nseeds) {
      unsigned long long s = atomicAdd(&sc->seed_next.v, 1ull);
      if (s < nseeds) {
        slot = s;
        return 1;
      }
    }
    seeds_done = true;
  }
  const unsigned long long t = atomicAdd(&sc->pop_cnt.v, 1ull);
  __threadfence();
  if (ld_volatile(sc->done.v)) return 0;
  long long t0 = clock64();
  unsigned long long last_prog = ld_volatile(sc->progress.v);
  unsigned ns = 32;
  const unsigned long long *seq = P.job_seq + (t & (P.job_ring - 1));
  for (uint32_t it = 0;; ++it) {
    unsigned long long r = ld_volatile(*seq);
    if (r == t + 1) {
      __threadfence();
      slot = t;
      atomicAdd(&sc->steals, 1ull);
      return 2;
    }
    if (r == (t | kSeqDone)) return 0;
    if ((it & 7) == 7) {
      if (ld_volatile(sc->done.v) || ld_volatile(sc->error)) return 0;
      unsigned long long pr = ld_volatile(sc->progress.v);
      if (pr != last_prog) {
        last_prog = pr;
        t0 = clock64();
      } else if (clock64() - t0 > P.timeout_cycles) {
        atomicOr(&sc->error, kErrTimeout);
        return 0;
      }
    }
    __nanosleep(ns);
    ns = min(ns * 2, 2048u);
  }
}

// Called by the whole warp once its task is finished.
__device__ void finish_task(const MatchArgs &P) {
  const uint32_t lane = threadIdx.x & 31;
  unsigned long long before = 0;
  if (lane == 0) before = atomicAdd(&P.sc->outstanding.v, ~0ull);
  before = __shfl_sync(kFull, before, 0);
  if (before != 1) return;
  // Last task of the launch: release every warp still waiting on a ticket.
  // Every position below push_cnt has been consumed (nothing is outstanding),
  // so the slot of each waiting ticket t is free and holds t; at most one
  // ticket per warp waits, far fewer than the ring's slots.
  unsigned long long lo = 0, hi = 0;
  if (lane == 0) {
    atomicExch(&P.sc->done.v, 1ull);
    __threadfence();
    hi = ld_volatile(P.sc->pop_cnt.v);
    lo = ld_volatile(P.sc->push_cnt.v);
  }
  lo = __shfl_sync(kFull, lo, 0);
  hi = __shfl_sync(kFull, hi, 0);
  for (unsigned long long t = lo + lane; t < hi; t += 32)
    atomicExch(&P.job_seq[t & (P.job_ring - 1)], t | kSeqDone);
}

// A task's search goes depth-first over batches: up to 32 partial embeddings
// of one level, a lane each, are expanded together.  E(l) is the expansion of
// the batch of level l (its partials fix positions 0..l) to level t = l + 1:
// each lane reads its partial's ranges of t's label in the runs of t's
// backward neighbours and takes the shortest as its pivot; the pivot ranges
// are laid end to end (a warp scan of their lengths) and scanned 32 entries at
// a time, each lane finding its entry's owner by a five-step search through
// the scan.  Survivors are appended to level t's buffer; 32 of them, or the
// rest when the ranges end, become the next batch.
//
// Bound by the warp's instructions and dependent loads, not by bandwidth (L2
// hit 94 %, DRAM idle).  One partial at a time, a level's set-up, descent and
// return were paid per candidate (about 2000 cycles each, half the matcher's
// time on queries of 8 to 12 vertices) and a chunk of one short range left most
// lanes idle; a batch pays them once for 32 and its chunks are full (31 of 32
// lanes, where 16 to 19 had an entry).  About 370 instructions a chunk, a
// quarter of them the search of the other ranges, at 0.6 issued a cycle (8
// warps a scheduler at 64 registers).  Matcher time of one batch, one B200: 64
// twelve-vertex queries x 32,768 updates on a hub-heavy 2^22-edge graph 51 ->
// 18 ms; 256 queries x 1021 updates on a 2^22-edge power-law graph 75 -> 42 ms;
// three queries x 4096 updates on a 2^24-edge one 86 -> 46 ms; one request of
// 512 updates against 64 queries 5.5 -> 2.6 ms.
//
// A level with several backward neighbours is scanned in two steps.  The
// graph's edge filter answers for the neighbours beside the pivot in one load
// each, where a search of a run takes 8 to 14 dependent ones, and most entries
// are turned away (on a 2^24-edge power-law graph 27 of 32): those that pass
// are gathered, and 32 of them searched together.  Three queries x 4096
// updates on that graph 44 -> 26 ms, 256 queries x 1021 updates 34 -> 24 ms;
// where most entries pass (a hub-heavy graph with 8 labels) it neither gains
// nor costs (15 ms).
//
// kLM: label-major runs with slot offsets (the engine's graph); otherwise plain
// id-sorted runs (the allocation-free entry point): a position's range is then
// the whole run and every entry's label is read.
//
// Shared memory of a warp (W = widest query): the batch's images F[W][32]
// (column k: the partial of lane k), up to kRows ranges per partial, the pivot
// per partial, 64 candidates (position in the ranges, id | owner << 27), and a
// buffer of 64 survivors per level (id | parent << 27; plain runs, whose ids may
// take all 32 bits, keep the parents behind the ids).
//
// Entries of a batch are counted in 32 bits: 32 ranges of an engine's graph hold
// fewer than 2^32 (its ids have 27 bits); of plain runs' partials those are
// taken whose ranges do.
constexpr uint32_t kPast = 0xFFFFFFFFu;  // no run is as long: a vertex has fewer neighbours than there are ids
// Partials together where the caller asks for small batches (DSM_OPT_PACK_MAX 0),
// which deal a search of few partials out sooner.  One at a time took longer on
// 256 queries x 1021 updates than the matcher without batches did (275 against
// 218 ms a batch and its undoing; two 167, four 108, eight 75, 32 49); four are
// no slower than it anywhere (three screened queries 1.9 -> 1.5 ms).
constexpr uint32_t kFew = 4;
constexpr uint32_t kRows = 3;  // backward neighbours with stored ranges; further ones are read when needed
template <bool kLM>
__host__ __device__ constexpr uint32_t warp_words(uint32_t W) {
  return W * 32 + kRows * 128 + 128 + 128 + (W > 3 ? W - 3 : 1) * (kLM ? 64 : 128);
}

template <bool kLM>
__device__ void run_task(const MatchArgs &P, const DevBatchEdges &bt, uint32_t nupd, uint32_t upd, uint32_t qo,
                         uint32_t depth, uint32_t lo, uint32_t hi, uint32_t fval, uint32_t *sm) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t(*const F)[32] = reinterpret_cast<uint32_t(*)[32]>(sm);
  uint4(*const rows)[32] = reinterpret_cast<uint4(*)[32]>(sm + P.W * 32);
  uint4 *const piv = reinterpret_cast<uint4 *>(sm + P.W * 32 + kRows * 128);
  uint2 *const cand = reinterpret_cast<uint2 *>(sm + P.W * 32 + kRows * 128 + 128);
  constexpr uint32_t kBuf = kLM ? 64 : 128;
  uint32_t(*const buf)[kBuf] = reinterpret_cast<uint32_t(*)[kBuf]>(sm + P.W * 32 + kRows * 128 + 256) - 2;  // from level 2
  // survivor i of level t: its image, and the lane of its partial below
  auto put = [&](uint32_t t, uint32_t i, uint2 x) {
    if constexpr (kLM) {
      buf[t][i] = x.x | (x.y << kIdBits);
    } else {
      buf[t][i] = x.x;
      buf[t][64 + i] = x.y;
    }
  };
  auto get = [&](uint32_t t, uint32_t i) -> uint2 {
    const uint32_t x = buf[t][i];
    if constexpr (kLM) return make_uint2(x & kIdMask, x >> kIdBits);
    else return make_uint2(x, buf[t][64 + i]);
  };
  const QDev &Q = P.qd[qo >> 8];
  const uint32_t nq = Q.nq;
  const OrderRec &R = P.orders[Q.order_base + (qo & 255)];
  // lane p: position p's backward neighbours, label and query vertex; lane k:
  // query vertex k's position
  const uint32_t q_vert = lane < 16 ? R.vert[lane] : 0;
  const uint32_t q_word = lane < 16 ? R.bn[lane] | (Q.label[q_vert & 15] << 16) | (q_vert << 21) |
                                          ((uint32_t)R.pos_of[lane] << 25)
                                    : 0u;
  const uint32_t tp = P.vtp[upd];
  const uint32_t *bitmap = Q.bitmap;
  const uint32_t seg = Q.local * nupd + upd;
  unsigned long long task_cnt = 0, work = 0;  // warp-uniform
  uint32_t alg = 0;                           // bytes, this lane's share since they were last added up
  // what the segment had left of its work limit when this task last looked
  // (at most 2^32 - 1): a task that alone exceeds it publishes at once, but for
  // a query with a listing budget, which the tuples listed until the heartbeat
  // count towards
  uint32_t work_left = 0xFFFFFFFFu;

  // Listing reserves slots in the result table; a query past its listing
  // budget reserves none (its count stays exact, the partial tuples are
  // dropped).  Survivors m hold w at position t, F's column k before it.
  auto emit = [&](uint32_t m, uint32_t w, uint32_t t, uint32_t k) {
    const uint32_t cnt = __popc(m);
    if (cnt == 0) return;
    task_cnt += cnt;
    if (!P.list) return;
    unsigned long long base = ~0ull;
    if (lane == 0) {
      bool ok = true;
      if (P.qlimit) ok = atomicAdd(&P.qlisted[Q.local], (unsigned long long)cnt) + cnt <= P.qlimit;
      if (ok) base = atomicAdd(&P.sc->out_count.v, (unsigned long long)cnt);
    }
    base = __shfl_sync(kFull, base, 0);
    if (base == ~0ull) return;
    const unsigned long long s = base + __popc(m & lanemask_lt());
    const bool wr = ((m >> lane) & 1u) && s < P.cap;
    if (wr) P.out_seg[s] = seg;
    for (uint32_t v = 0; v < nq; ++v) {
      const uint32_t p = __shfl_sync(kFull, q_word, v) >> 25;
      if (wr) P.out_tup[s * P.W + v] = p == t ? w : F[p][k];
    }
    if (wr) alg += 4 * (nq + 1);
  };

  // Work limit (P.work_limit > 0): `work` counts the valid partial
  // embeddings of 3 or more positions this task generated (embeddings
  // included).  The total of a (query, update) segment does not depend on
  // scheduling, so "the segment's total reached the limit" is deterministic:
  // whoever's addition crosses it sets bit 63 of the segment's count, and the
  // segment's tasks stop (its count is then partial, marked by that bit).
  auto publish_work = [&]() -> bool {  // true: the segment is over its limit
    uint32_t left = 0;
    if (lane == 0) {
      const unsigned long long before = work ? atomicAdd(&P.seg_work[seg], work) : ld_volatile(P.seg_work[seg]);
      if (before + work < P.work_limit) left = (uint32_t)min(P.work_limit - before - work, 0xFFFFFFFFull);
      else if (work && before < P.work_limit) atomicOr(&P.seg_count[seg], kCountIncomplete);
    }
    work = 0;
    work_left = __shfl_sync(kFull, left, 0);
    return work_left == 0;
  };

  auto add_bytes = [&]() {
    const uint32_t a0 = __reduce_add_sync(kFull, alg & 0xFFFFu), a1 = __reduce_add_sync(kFull, alg >> 16);
    if (lane == 0) atomicAdd(&P.sc->alg_bytes, ((unsigned long long)a1 << 16) + a0);
    alg = 0;
  };
  auto flush = [&]() {
    if (P.work_limit && work) publish_work();
    if (lane == 0 && task_cnt) {
      atomicAdd(&P.seg_count[seg], task_cnt);
      atomicAdd(&P.sc->matches, task_cnt);
    }
    add_bytes();
  };

  __syncwarp();  // the last task's reads of the warp's shared memory are done
  for (uint32_t p = 0; p < depth; ++p) F[p][lane] = __shfl_sync(kFull, fval, p);
  __syncwarp();
  if (depth >= nq) {  // a one-edge query: the seed is the embedding
    emit(1u, 0, 0xFFFFFFFFu, 0);
    flush();
    return;
  }
  if (P.work_limit && publish_work()) return;  // a segment already over its limit

  // the expansion at hand, E(l) to level t = l + 1 (warp-uniform): next and
  // last entry of the ranges laid end to end, partials of the batch, survivors
  // in t's buffer; t's backward neighbours, label, and the earlier positions
  // with that label
  uint32_t l = depth - 1, c = 0, e = 0, nb = 1, cnt = 0, t_bn = 0, t_lab = 0, t_same = 0;
  uint32_t incl = 0, len = 0;               // lane k: scan of the pivot ranges, this partial's
  // E(lane), parked while deeper ones run: lv_n = nb | cnt << 8 | partials
  // whose range is not begun << 16
  uint32_t lv_c = 0, lv_e = 0, lv_n = 0;
  const uint32_t most = P.pack_max ? 32u : kFew;  // partials expanded together

  // The ranges of E(l)'s partials (F holds the batch); returns their total.
  // Plain runs: may make the batch smaller, so that the total fits.
  auto setup = [&]() -> uint32_t {
    const uint32_t tw = __shfl_sync(kFull, q_word, l + 1);
    t_bn = tw & 0xFFFFu;
    t_lab = (tw >> 16) & 31u;
    t_same = __ballot_sync(kFull, lane <= l && ((q_word >> 16) & 31u) == t_lab);
    uint32_t best = 0xFFFFFFFFu, pr = 0, pa = 0, poff = 0, r = 0;
    for (uint32_t bits = t_bn; bits; bits &= bits - 1, ++r) {
      uint32_t a = 0, b = 0, off = 0, touched = 0;
      if constexpr (kLM) {
        if (lane < nb && t_lab < P.g.nlt) {
          const uint32_t x = F[__ffs(bits) - 1][lane];
          const uint32_t *o = P.g.loff + (size_t)x * (P.g.nlt + 1) + t_lab;
          a = o[0];
          b = o[1];
          off = P.g.adj[x].x;
          touched = P.g.lab[x] >> 31;
          alg += 8;
        }
      } else if (lane < nb) {
        const uint2 x = P.g.adj[F[__ffs(bits) - 1][lane]];
        off = x.x;
        b = x.y;
      }
      if (r < kRows) rows[r][lane] = make_uint4(off, a, b, touched);
      if (b - a < best) {
        best = b - a;
        pr = r;
        pa = a;
        poff = off;
      }
    }
    len = lane < nb ? best : 0u;
    incl = len;
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
      const uint32_t x = __shfl_up_sync(kFull, incl, d);
      if (lane >= d) incl = kLM || incl + x >= x ? incl + x : kPast;
    }
    if constexpr (!kLM) {  // the partials from which on the sum does not fit stay in the buffer (the first fits)
      const uint32_t fit = __popc(__ballot_sync(kFull, incl != kPast));
      if (fit < nb) {
        nb = fit;
        incl = min(incl, __shfl_sync(kFull, incl, nb - 1));
        if (lane >= nb) len = 0;
      }
    }
    const uint64_t start = (uint64_t)poff * 4 + pa - (incl - len);  // entry i of the scan is arena[start + i]
    piv[lane] = make_uint4((uint32_t)start, (uint32_t)(start >> 32), pr, pa);
    __syncwarp();
    return __shfl_sync(kFull, incl, 31);
  };

  auto park = [&]() {
    const uint32_t excl = incl - len;
    const uint32_t todo = __popc(__ballot_sync(kFull, len && excl >= c && excl < e));
    if (lane == l) {
      lv_c = c;
      lv_e = e;
      lv_n = nb | (cnt << 8) | (todo << 16);
    }
  };

  // F for the batch of level l from the buffers (levels depth..l).
  auto rebuild = [&]() {
    __syncwarp();
    uint32_t k = lane;
    for (uint32_t j = l; j >= depth; --j) {
      const uint2 x = get(j, k);
      F[j][lane] = x.x;
      k = x.y & 31;
    }
    __syncwarp();
  };

  // Counting, E(nq - 2): a last position with one backward neighbour x has as
  // many images as x's range holds, less those whose edge is not live and the
  // images of earlier positions with its label that lie in it; no entry is
  // read.  (A candidate filter's bitmap, or a slot that several labels share,
  // would have to be asked for every entry.)
  auto counts_only = [&]() -> bool {
    if (!P.list) return true;
    if (!P.qlimit) return false;  // over its listing budget a query is only counted
    uint32_t over = 0;
    if (lane == 0) over = ld_volatile(P.qlisted[Q.local]) > P.qlimit;
    return __shfl_sync(kFull, over, 0) != 0;
  };
  bool cnt_only = !bitmap && counts_only();
  auto leaf_count = [&]() {
    const uint32_t j = __ffs(t_bn) - 1, j_bn = __shfl_sync(kFull, q_word, j) & 0xFFFFu;
    const uint4 row = rows[0][lane];
    const uint32_t x = F[j][lane];
    uint32_t gone = 0;
    if (len && row.w && may_change(bt, x, slot_key(t_lab))) gone = dead_entries(bt, x, t_lab, tp, &P.sc->progress.v);
    for (uint32_t same = t_same & ~(1u << j); same; same &= same - 1) {
      const uint32_t i = __ffs(same) - 1, i_bn = __shfl_sync(kFull, q_word, i) & 0xFFFFu;
      if (((j_bn >> i) | (i_bn >> j)) & 1u) {
        ++gone;  // a live neighbour of x: the query has that edge
      } else if (len > gone) {
        const uint32_t y = F[i][lane];
        if (run_has(P.g.arena + (uint64_t)row.x * 4 + row.y, len, pack_entry(t_lab, y)) &&
            !(row.w && may_change(bt, x, y) && !edge_live(bt, x, y, tp)))
          ++gone;
      }
    }
    uint32_t n = len > gone ? len - gone : 0u;
    const unsigned long long sum =
        (unsigned long long)__reduce_add_sync(kFull, n & 0xFFFFu) + ((unsigned long long)__reduce_add_sync(kFull, n >> 16) << 16);
    work += sum;
    task_cnt += sum;
  };

  // The survivors m of E(l) (lane: image w, owner k) as rows of l + 2 fixed
  // positions.  One reservation per chunk, all or nothing (a bounded
  // compare-and-swap loop); false: no room, nothing written.
  auto write_rows = [&](uint32_t m, uint32_t w, uint32_t k) -> bool {
    const uint32_t n = __popc(m);
    unsigned long long base = ~0ull;
    if (lane == 0) {
      unsigned long long cur = ld_volatile(*P.rows_cnt);
      for (int tries = 0; tries < 64 && cur + n <= P.rows_cap; ++tries) {
        const unsigned long long prev = atomicCAS(P.rows_cnt, cur, cur + n);
        if (prev == cur) {
          base = cur;
          break;
        }
        cur = prev;
      }
    }
    base = __shfl_sync(kFull, base, 0);
    if (base == ~0ull) return false;
    if ((m >> lane) & 1u) {
      uint32_t *rec = reinterpret_cast<uint32_t *>(P.rows_out + base + __popc(m & lanemask_lt()));
      __stcg(rec, upd);
      __stcg(rec + 1, qo);
      __stcg(rec + 2, l + 2);
      for (uint32_t j = 0; j <= l; ++j) __stcg(rec + 8 + j, F[j][k]);
      __stcg(rec + 9 + l, w);
    }
    return true;
  };

  // Whether E(l), just set up, is counted without a scan.  256 entries: eight
  // chunks take longer than the searches for images in the range (from 1 on,
  // screened 8-vertex queries lost 5 to 15 %, from 256 on none; 256 queries x
  // 1021 updates gain 10 % at any bound up to 512).
  auto leaf = [&]() -> bool {
    return kLM && cnt_only && l + 2 == nq && e >= 256 && (t_bn & (t_bn - 1)) == 0 && t_lab < 31;
  };

  e = setup();
  if (hi) {  // a donated part [lo, hi) of the one partial's pivot range
    const uint32_t pa = piv[0].w;
    c = lo - pa;
    e = min(e, hi - pa);
  } else if (leaf()) {
    leaf_count();
    c = e;
  }
  uint32_t hb = 0;     // chunks since the last heartbeat
  // tuples count towards a listing budget until the search is found over its
  // limit: heartbeats by partial embeddings too
  const bool beat = P.work_limit && P.qlimit && P.list;
  int32_t dticks = 0;  // chunks since the last donation check (below zero: none for a while)
  uint32_t nc = 0;  // candidates that passed the edge filter
  while (true) {
    if (cnt < most && (c < e || nc)) {
      const uint32_t t = l + 1;
      const bool two = kLM && P.g.flt && (t_bn & (t_bn - 1));
      bool ok = false, test = true;
      uint32_t k = 0, w = 0;
      if (!two || (nc < 32 && c < e)) {  // a chunk of the ranges
        const uint32_t pos = c + lane;
        ok = lane < e - c;
#pragma unroll
        for (uint32_t d = 16; d; d >>= 1) {  // the owner: the first lane with incl > pos
          const uint32_t v = __shfl_sync(kFull, incl, k + d - 1);
          if (v <= pos) k += d;
        }
        const uint4 pv = piv[k];
        if (ok) {
          w = P.g.arena[((uint64_t)pv.y << 32 | pv.x) + pos];
          if constexpr (kLM) w &= kIdMask;
          alg += 4;
        }
        c = e - c > 32 ? c + 32 : e;
        if (two) {
          uint32_t r = 0;
          for (uint32_t bits = t_bn; bits; bits &= bits - 1, ++r)
            if (ok && r != pv.z) {
              ok = may_have(P.g, F[__ffs(bits) - 1][k], w);
              alg += 4;
            }
          const uint32_t m = __ballot_sync(kFull, ok);
          if (ok) cand[nc + __popc(m & lanemask_lt())] = make_uint2(pos, w | (k << kIdBits));
          nc += __popc(m);
          test = nc >= 32 || (c >= e && nc);
          __syncwarp();
        }
      }
      if (two && test) {  // up to 32 of those that passed
        const uint32_t n = min(nc, 32u);
        const uint2 x = cand[lane], y = cand[32 + lane];
        __syncwarp();
        if (32 + lane < nc) cand[lane] = y;
        __syncwarp();  // the descent reads the first of the rest, the next chunk writes behind them
        ok = lane < n;
        w = x.y & kIdMask;
        k = ok ? x.y >> kIdBits : 0u;
        nc -= n;
      }
      if (test) {
        const uint32_t en = kLM ? (t_lab << kIdBits) | w : w;
        if (!kLM || t_lab >= 31)  // plain runs hold every label, slot 31 every label >= 31
          ok = ok && ((P.g.lab[w] & kLabelMask) == t_lab);
        // injectivity: only earlier positions with the same label can hold w
        for (uint32_t same = t_same; same; same &= same - 1) ok = ok && w != F[__ffs(same) - 1][k];
        if (bitmap) {
          const uint32_t qv = (__shfl_sync(kFull, q_word, t) >> 21) & 15u;
          ok = ok && ((bitmap[(size_t)qv * Q.col_len + (w >> 5)] >> (w & 31)) & 1u);
        }
        uint32_t r = 0;
        for (uint32_t bits = t_bn; bits; bits &= bits - 1, ++r) {
          if (!ok) continue;
          const uint32_t j = __ffs(bits) - 1;
          uint4 row;
          if (r < kRows) {
            row = rows[r][k];
          } else {
            const uint32_t x = F[j][k];
            if constexpr (kLM) {
              const uint32_t *o = P.g.loff + (size_t)x * (P.g.nlt + 1) + t_lab;
              row = make_uint4(P.g.adj[x].x, o[0], o[1], P.g.lab[x] >> 31);
            } else {
              const uint2 a = P.g.adj[x];
              row = make_uint4(a.x, 0, a.y, 0);
            }
          }
          if (r != piv[k].z) {
            ok = run_has(P.g.arena + (uint64_t)row.x * 4 + row.y, row.z - row.y, en);
            alg += 4;
          }
          // liveness: only edges of a touched vertex can have changed, and of
          // those the filter turns away all that the batch does not change
          if (kLM && ok && row.w) {
            const uint32_t x = F[j][k];
            if (may_change(bt, x, w)) ok = edge_live(bt, x, w, tp);
          }
        }
        const uint32_t m = __ballot_sync(kFull, ok);
        const uint32_t ns = __popc(m);
        work += ns;
        if (t == nq - 1) {
          emit(m, w, t, k);
        } else if (m && !(P.bfs_stop == t + 1 && write_rows(m, w, k))) {
          if (ok) put(t, cnt + __popc(m & lanemask_lt()), make_uint2(w, k));
          cnt += ns;
        }
      }
      ++hb;
      ++dticks;
      if (P.work_limit && work >= work_left && (!P.qlimit || cnt_only)) {
        if (publish_work()) break;
      }
      if (hb >= 64 || (beat && work >= kListBeat)) {
        hb = 0;
        unsigned int err = 0;
        if (lane == 0) {
          atomicAdd(&P.sc->progress.v, 1ull);
          err = ld_volatile(P.sc->error);
        }
        if (__shfl_sync(kFull, err, 0)) break;
        if (__any_sync(kFull, alg >> 31)) add_bytes();  // a lane reads far less than 2^31 bytes in 64 chunks
        if (P.work_limit && publish_work()) break;
        if (P.qlimit && !cnt_only) cnt_only = !bitmap && counts_only();
      }
      if (P.donate && dticks >= 8) {
        dticks = 0;
        unsigned long long h = 0;
        if (lane == 0) {
          const unsigned long long pc = ld_volatile(P.sc->pop_cnt.v), pu = ld_volatile(P.sc->push_cnt.v);
          h = pc > pu ? pc - pu : 0;
        }
        h = __shfl_sync(kFull, h, 0);
        if (h > 0) {
          const uint32_t split_min = P.split_min > 64 ? P.split_min : (P.split_min ? 64u : 128u);
          const uint32_t dd = P.donate_depth ? min(P.donate_depth, 4u) : 2u;
          park();  // so that every expansion reads alike
          // the shallowest expansion with a substantial piece of work: waiting
          // survivors with dd or more levels below them, partials not begun,
          // or a long rest of one range
          const uint32_t above = __shfl_down_sync(kFull, lv_n, 1) & 0xFFu;  // its survivors already descended into
          const uint32_t wait = ((lv_n >> 8) & 0xFFu) - (lane < l ? above : 0u);
          const bool has = lane + 1 >= depth && lane <= l &&
                           ((wait && lane + 1 + dd < nq) ||
                            ((lv_n >> 16) && lane + dd < nq) || lv_e - lv_c >= split_min);
          const uint32_t hm = __ballot_sync(kFull, has);
          if (hm) {
            __syncwarp();  // the survivors in the buffers are visible to every lane
            const uint32_t l0 = l, i = __ffs(hm) - 1;
            const uint32_t wi = __shfl_sync(kFull, wait, i);
            if (i != l) {
              l = i;
              nb = __shfl_sync(kFull, lv_n, i) & 0xFFu;
              rebuild();
              setup();
            }
            const uint32_t ci = __shfl_sync(kFull, lv_c, i), ei = __shfl_sync(kFull, lv_e, i);
            uint32_t ni = (__shfl_sync(kFull, lv_n, i) >> 8) & 0xFFu, todo = __shfl_sync(kFull, lv_n, i) >> 16, ecut = ei;
            // this lane's job, if any: column jk of F, image jw of position
            // i + 1 (jdepth = i + 2) or a range of it
            bool mine = false;
            uint32_t jk = 0, jw = 0, jdepth = i + 1, jlo = 0, jhi = 0, jobs = 0;
            if (wi && i + 1 + dd < nq) {
              jobs = min(wi, (uint32_t)min(h, 32ull));
              mine = lane < jobs;
              const uint2 x = mine ? get(i + 1, ni - jobs + lane) : make_uint2(0, 0);
              jk = x.y;
              jw = x.x;
              jdepth = i + 2;
            } else {
              const uint32_t excl = incl - len;
              uint32_t um = i + dd < nq ? __ballot_sync(kFull, len && excl >= ci && excl < ei) : 0u;
              if (um) {  // whole partials, the last ones
                jobs = min((uint32_t)__popc(um), (uint32_t)min(h, 32ull));
                for (uint32_t x = __popc(um); x > jobs; --x) um &= um - 1;
                mine = (um >> lane) & 1u;
                jk = lane;
                if (incl > ei) {  // the last one without what was cut off before
                  jlo = piv[lane].w;
                  jhi = jlo + (ei - excl);
                }
                ecut = __shfl_sync(kFull, excl, __ffs(um) - 1);
                todo -= jobs;
              } else if (ei - ci >= split_min) {
                // half of what is left, a job for each partial it reaches into
                // (the last ones, when fewer warps wait)
                uint32_t mid = ci + (((ei - ci) / 2 + 31) & ~31u);
                um = __ballot_sync(kFull, len && incl > mid && excl < ei);
                jobs = min((uint32_t)__popc(um), (uint32_t)min(h, 32ull));
                for (uint32_t x = __popc(um); x > jobs; --x) um &= um - 1;
                if (um) {
                  mine = (um >> lane) & 1u;
                  jk = lane;
                  mid = max(mid, __shfl_sync(kFull, excl, __ffs(um) - 1));
                  jlo = piv[lane].w + (max(excl, mid) - excl);
                  jhi = piv[lane].w + (min(incl, ei) - excl);
                  ecut = mid;
                  todo = __popc(__ballot_sync(kFull, len && excl >= ci && excl < ecut));
                }
              }
            }
            unsigned long long s0 = 0;
            uint32_t okr = 0;
            const unsigned long long rmask = P.job_ring - 1;
            if (lane == 0 && jobs) {
              // jobs <= waiting warps, so positions stay within one warp's worth
              // of reservations per donor of pop_cnt: the slot of position p
              // was last used by position p - ring, consumed long ago; wait
              // (bounded) until its consumer has released it
              atomicAdd(&P.sc->outstanding.v, (unsigned long long)jobs);
              s0 = atomicAdd(&P.sc->push_cnt.v, (unsigned long long)jobs);
              atomicAdd(&P.sc->donations, (unsigned long long)jobs);
              okr = 1;
              const long long tw = clock64();
              for (uint32_t x = 0; x < jobs && okr; ++x)
                while (ld_volatile(P.job_seq[(s0 + x) & rmask]) != s0 + x) {
                  if (clock64() - tw > P.timeout_cycles) {
                    atomicOr(&P.sc->error, kErrTimeout);
                    okr = 0;
                    break;
                  }
                  __nanosleep(64);
                }
            }
            okr = __shfl_sync(kFull, okr, 0);
            s0 = __shfl_sync(kFull, s0, 0);
            if (okr) {
              const uint32_t mm = __ballot_sync(kFull, mine);
              if (mine) {
                const unsigned long long at = s0 + __popc(mm & lanemask_lt());
                uint32_t *rec = reinterpret_cast<uint32_t *>(P.jobs + (at & rmask));
                __stcg(rec, upd);
                __stcg(rec + 1, qo);
                __stcg(rec + 2, jdepth);
                __stcg(rec + 3, jlo);
                __stcg(rec + 4, jhi);
                for (uint32_t j = 0; j <= i; ++j) __stcg(rec + 8 + j, F[j][jk]);
                if (jdepth == i + 2) __stcg(rec + 9 + i, jw);
                __threadfence();
                atomicExch(&P.job_seq[at & rmask], at + 1);
              }
              if (jdepth == i + 2) ni -= jobs;
              if (lane == i) {
                lv_e = ecut;
                lv_n = (lv_n & 0xFFu) | (ni << 8) | (todo << 16);
              }
            } else {
              dticks = -8;  // nothing to give, or a failed wait
            }
            if (i != l0) {
              l = l0;
              nb = __shfl_sync(kFull, lv_n, l) & 0xFFu;
              rebuild();
              setup();
            }
            e = __shfl_sync(kFull, lv_e, l);
            cnt = (__shfl_sync(kFull, lv_n, l) >> 8) & 0xFFu;
          }
        }
      }
      continue;
    }
    if (cnt) {  // descend: up to 32 survivors become the next batch
      if (nc) {  // candidates not tested yet are read again
        c = cand[0].x;
        nc = 0;
      }
      park();
      __syncwarp();
      nb = min(cnt, most);
      const uint2 x = get(l + 1, lane < nb ? lane : 0);
      for (uint32_t j = depth; j <= l; ++j) {
        const uint32_t v = F[j][x.y];
        __syncwarp();
        F[j][lane] = v;
      }
      ++l;
      F[l][lane] = x.x;
      __syncwarp();
      c = 0;
      cnt = 0;
      e = setup();
      if (leaf()) {
        leaf_count();
        c = e;
        ++hb;
        if (P.work_limit && work >= work_left) {
          if (publish_work()) break;
        }
      }
      continue;
    }
    if (l + 1 == depth) break;
    // back to E(l - 1): its buffer without the batch just done
    const uint32_t done = nb;
    --l;
    c = __shfl_sync(kFull, lv_c, l);
    e = __shfl_sync(kFull, lv_e, l);
    nb = __shfl_sync(kFull, lv_n, l);
    cnt = ((nb >> 8) & 0xFFu) - done;
    nb &= 0xFFu;
    if (cnt || c < e) {
      __syncwarp();
      uint2 y[2];
#pragma unroll
      for (uint32_t h = 0; h < 2; ++h)
        y[h] = lane + 32 * h < cnt ? get(l + 1, done + lane + 32 * h) : make_uint2(0, 0);
      __syncwarp();
#pragma unroll
      for (uint32_t h = 0; h < 2; ++h)
        if (lane + 32 * h < cnt) put(l + 1, lane + 32 * h, y[h]);
      rebuild();
      if (c < e) setup();
    }
  }
  flush();
}

// phantom = 1 adds one outstanding task that nothing finishes (a test of the
// bounded waits: the launch then ends only through their timeouts).
__global__ void k_sched_init(Sched *sc, const BatchHdr *hdr, unsigned long long *job_seq, uint32_t job_ring,
                             uint32_t phantom) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned long long seed_cap = hdr ? hdr->seed_cap : ~0ull;  // no header: tasks are rows
  for (uint32_t s = i; s < job_ring; s += gridDim.x * blockDim.x) job_seq[s] = s;
  if (i == 0) {
    unsigned long long n = sc->nseeds;
    if (n > seed_cap) {
      sc->nseeds = n = seed_cap;
      atomicOr(&sc->error, kErrSeeds);
    }
    sc->outstanding.v = n + phantom;
    sc->done.v = (n + phantom == 0) ? 1ull : 0ull;
  }
}

template <bool kLM>
__global__ void __launch_bounds__(256, 4) k_match(MatchArgs P) {
  extern __shared__ __align__(16) uint32_t smem[];
  const uint32_t lane = threadIdx.x & 31;
  if (*P.abort_flag & kErrArena) return;  // the batch was refused before its insert
  // an earlier launch of this batch failed (one read, the same for the warp:
  // the word can change while the kernel runs)
  if (__shfl_sync(kFull, lane == 0 ? ld_volatile(P.sc->error) : 0u, 0)) return;
  const uint32_t nupd = P.hdr->n;
  const DevBatchEdges bt{P.bt.bkey, P.bt.binfo, P.bt.bloom, P.bt.table, P.bt.dkey, P.hdr->m, P.hdr->bloom_mask};
  bool seeds_done = false;
  while (true) {
    uint32_t kind = 0;
    unsigned long long slot = 0;
    if (lane == 0) kind = acquire(P, slot, seeds_done);
    kind = __shfl_sync(kFull, kind, 0);
    if (kind == 0) break;
    slot = __shfl_sync(kFull, slot, 0);
    uint32_t upd, qo, depth, lo = 0, hi = 0, fval = 0;
    if (kind == 1 && P.rows_in) {  // a row written by the previous launch
      const uint32_t word = __ldcg(reinterpret_cast<const uint32_t *>(P.rows_in + slot) + lane);
      upd = __shfl_sync(kFull, word, 0);
      qo = __shfl_sync(kFull, word, 1);
      depth = __shfl_sync(kFull, word, 2);
      fval = __shfl_sync(kFull, word, (lane + 8) & 31);
    } else if (kind == 1) {
      uint4 s = P.seeds[slot];
      upd = s.x;
      qo = s.y;
      depth = 2;
      fval = lane == 0 ? s.z : (lane == 1 ? s.w : 0u);
    } else {
      const uint32_t *rec = reinterpret_cast<const uint32_t *>(P.jobs + (slot & (P.job_ring - 1)));
      uint32_t word = __ldcg(rec + lane);
      __syncwarp();
      if (lane == 0) {  // the slot is free for position slot + ring
        __threadfence();
        atomicExch(&P.job_seq[slot & (P.job_ring - 1)], slot + P.job_ring);
      }
      upd = __shfl_sync(kFull, word, 0);
      qo = __shfl_sync(kFull, word, 1);
      depth = __shfl_sync(kFull, word, 2);
      lo = __shfl_sync(kFull, word, 3);
      hi = __shfl_sync(kFull, word, 4);
      fval = __shfl_sync(kFull, word, (lane + 8) & 31);
    }
    run_task<kLM>(P, bt, nupd, upd, qo, depth, lo, hi, fval, smem + (threadIdx.x >> 5) * warp_words<kLM>(P.W));
    finish_task(P);
  }
}

}  // namespace

__global__ void k_rows_arm(Sched *sc, const unsigned long long *rows_cnt, unsigned long long rows_cap) {
  sc->seeds = sc->nseeds;  // the seed table's count, for a rerun from the seeds
  sc->seed_next.v = 0;
  sc->push_cnt.v = 0;
  sc->pop_cnt.v = 0;
  sc->done.v = 0;
  sc->outstanding.v = 0;
  sc->nseeds = min(*rows_cnt, rows_cap);
}

void launch_rows_arm(Sched *sc, const unsigned long long *rows_cnt, unsigned long long rows_cap, cudaStream_t s) {
  k_rows_arm<<<1, 1, 0, s>>>(sc, rows_cnt, rows_cap);
}

void launch_sched_init(Sched *sc, const BatchHdr *hdr, unsigned long long *job_seq, uint32_t job_ring,
                       cudaStream_t s, uint32_t phantom) {
  k_sched_init<<<(job_ring + 255) / 256, 256, 0, s>>>(sc, hdr, job_seq, job_ring, phantom);
}

namespace {

// Shared memory of a block for queries of up to W vertices.
template <bool kLM>
constexpr int match_smem(uint32_t W) {
  return 8 * 4 * (int)warp_words<kLM>(W);
}

}  // namespace

cudaError_t match_prepare() {
  const cudaError_t e = cudaFuncSetAttribute(k_match<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             match_smem<true>(kMaxWidth));
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(k_match<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              match_smem<false>(kMaxWidth));
}

void launch_match(const MatchArgs &a, int blocks, cudaStream_t s) {
  if (a.g.loff) k_match<true><<<blocks, 256, match_smem<true>(a.W), s>>>(a);
  else k_match<false><<<blocks, 256, match_smem<false>(a.W), s>>>(a);
}

int match_max_blocks_per_sm(uint32_t width) {
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_match<true>, 256, match_smem<true>(width));
  return n;
}

}  // namespace dsm
