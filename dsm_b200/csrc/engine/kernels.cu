// Kernels of the batch pipeline around the matcher: edge state of a batch,
// in-place adjacency merge / removal, and seeding.
#include "kernels.cuh"

namespace dsm {

namespace {

template <class T>
__device__ __forceinline__ T ld_volatile(const T &x) {
  return *(const volatile T *)&x;
}

// Is {a, b} in the (label-major) graph: b's entry in the shorter of the two runs.
__device__ __forceinline__ bool has_edge(const DevGraph &g, uint32_t a, uint32_t b) {
  uint2 aa = g.adj[a], bb = g.adj[b];
  if (bb.y < aa.y) {
    uint2 t = aa;
    aa = bb;
    bb = t;
    uint32_t x = a;
    a = b;
    b = x;
  }
  const uint32_t key = pack_entry(g.lab[b] & kLabelMask, b);
  const uint32_t *l = adj_list(g, aa);
  uint32_t p = lower_bound_u32(l, aa.y, key);
  return p < aa.y && l[p] == key;
}

// ---------------------------------------------------------------------------
// Edge state of a batch
// ---------------------------------------------------------------------------
__global__ void k_edge_state(EdgeStateArgs A) {
  const uint32_t M = A.hdr->m;
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < M; j += gridDim.x * blockDim.x) {
  unsigned long long key = A.bkey[j];
  if (j > 0 && A.bkey[j - 1] == key) continue;  // not a group head
  uint32_t a = (uint32_t)(key >> 32), b = (uint32_t)key;
  bool init = has_edge(A.g, a, b);
  bool state = init, inserted = false, any_change = false;
  uint32_t e = j;
  for (; e < M && A.bkey[e] == key; ++e) {
    uint32_t i = A.bidx[e];
    uint32_t op = A.upd[i].x ? 1u : 0u;
    bool noop = op ? state : !state;
    A.binfo[e] = i | (op << 30) | ((uint32_t)init << 31);
    if (noop) {
      A.vtp[i] = kNoView;
    } else {
      any_change = true;
      A.vtp[i] = op ? i + 1 : i;  // insert: graph after it; delete: graph before it
      if (op) inserted = true;
    }
    state = op;
  }
  uint8_t flag = 0;
  if (!init && inserted) {
    flag |= 1;  // must join the union graph now
    if (A.g.flt) {
      uint32_t word;
      const uint32_t bits = bloom_bits(a, b, A.g.flt_mask, word);
      atomicOr(&A.g.flt[word], bits);
    }
  }
  if (!state && (init || inserted)) flag |= 2;  // must leave it after matching
  for (uint32_t k = j; k < e; ++k) A.gflag[k] = flag;
  if (any_change) {
    atomicOr(&A.g.lab[a], kTouchBit);
    atomicOr(&A.g.lab[b], kTouchBit);
    uint32_t word;
    const uint32_t bmask = A.hdr->bloom_mask;
    uint32_t bits = bloom_bits(a, b, bmask, word);
    atomicOr(&A.bloom[word], bits);
    bits = bloom_bits(a, slot_key(label_slot(A.g.lab[b] & kLabelMask)), bmask, word);
    atomicOr(&A.bloom[word], bits);
    bits = bloom_bits(b, slot_key(label_slot(A.g.lab[a] & kLabelMask)), bmask, word);
    atomicOr(&A.bloom[word], bits);
    // at most half of the slots are ever taken, so a free one is found
    const uint32_t mask = bmask >> 1;
    for (uint32_t sl = table_slot(key, mask); atomicCAS(&A.table[sl], 0u, j + 1) != 0u; sl = (sl + 1) & mask) {
    }
  }
  }
}

__device__ __forceinline__ uint8_t group_flag(const AdjUpdateArgs &A, uint32_t M, uint32_t x, uint32_t y) {
  unsigned long long key = canon_key(x, y);
  uint32_t lo = 0, hi = M;
  while (lo < hi) {
    uint32_t mid = (lo + hi) >> 1;
    if (A.bkey[mid] < key) lo = mid + 1; else hi = mid;
  }
  return (lo < M && A.bkey[lo] == key) ? A.gflag[lo] : 0;
}

// Compacts the entries of source group [s, e) selected by `want` (and, for
// inserts, not yet in the run) into dsel[s..s+k), in entry order.  Returns k.
// dkey holds x << 32 | entry of the neighbour, sorted.
__device__ uint32_t select_group(const AdjUpdateArgs &A, uint32_t M, uint32_t s, uint32_t e, uint32_t x,
                                 uint8_t want, bool skip_present, const uint32_t *L, uint32_t d) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t k = 0;
  for (uint32_t base = s; base < e; base += 32) {
    uint32_t j = base + lane;
    bool sel = false;
    uint32_t y = 0;
    if (j < e) {
      unsigned long long key = A.dkey[j];
      y = (uint32_t)key;
      bool first = (j == s) || (A.dkey[j - 1] != key);
      sel = first && (group_flag(A, M, x, y & kIdMask) & want);
      if (sel && skip_present) {
        uint32_t p = lower_bound_u32(L, d, y);
        sel = !(p < d && L[p] == y);
      }
    }
    uint32_t m = __ballot_sync(kFull, sel);
    if (sel) A.dsel[s + k + __popc(m & lanemask_lt())] = y;
    k += __popc(m);
  }
  __syncwarp();
  return k;
}

// A run's rewrite, by T threads: one warp (T = 32), or the whole block
// (T = 256) from kLongRun entries on.  Each entry of the run moves by the
// number of inserted (or removed) entries below it, found by a search of
// those few, so entries move independently, four a thread and 4 T at a time;
// the entries below the first change stay where they are and are not read.
// The warp-per-run merge that this replaces took 32 entries a step, each
// through a search of both lists: a hub of 10^5 entries held up the launch
// (512 updates on 2^20 vertices, 2^24 edges (R-MAT): insert 1002 -> 57 us,
// delete 932 -> 54 us; 32,768 updates on a hub-heavy 2^22-edge graph: update
// and marks 550 -> 220 us).  2048: a warp then takes 16 steps at most, and a
// block has two tiles to share.
constexpr uint32_t kLongRun = 2048;

template <uint32_t T>
__device__ __forceinline__ void sync_threads() {
  if constexpr (T == 32) __syncwarp();
  else __syncthreads();
}

// Merges N (k >= 1 entries, sorted, not in L) into the sorted run L (d
// entries) at out[0, d + k); out is L itself or a run that does not overlap
// it.  In place (k is then a fraction of d) the tiles go from the top down: a
// tile is read before it is written, and writes nothing below its own entries;
// the thread with the entry above them writes the new entries of a gap.  Into
// another run, where k may be many times d, every entry of both finds its place
// by itself (500,000 neighbours for a vertex of few, so in few gaps: the update
// 110 -> 91 ms; the rest is their selection by one warp).
template <uint32_t T>
__device__ void insert_run(const uint32_t *L, uint32_t d, const uint32_t *N, uint32_t k, uint32_t *out, uint32_t t) {
  if (out != L) {
    for (uint32_t r = t; r < k; r += T) out[r + lower_bound_u32(L, d, N[r])] = N[r];
    for (uint32_t b = 4 * t; b < d; b += 4 * T) {
      const uint4 q = *reinterpret_cast<const uint4 *>(L + b);
      const uint32_t v[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (uint32_t j = 0; j < 4; ++j)
        if (b + j < d) out[b + j + lower_bound_u32(N, k, v[j])] = v[j];
    }
    return;
  }
  const uint32_t first = lower_bound_u32(L, d, N[0]) & ~3u;
  if (d == first) {  // nothing moves: N follows the run (first = d only when d is a multiple of 4)
    for (uint32_t r = t; r < k; r += T) out[d + r] = N[r];
    return;
  }
  for (uint32_t tile = (d - first - 1) / (4 * T) + 1; tile-- > 0;) {
    const uint32_t b = first + tile * 4 * T + 4 * t;
    uint32_t v[4] = {0, 0, 0, 0}, prev = 0;
    if (b < d) {
      const uint4 q = *reinterpret_cast<const uint4 *>(L + b);
      v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
      if (b) prev = L[b - 1];
    }
    sync_threads<T>();
    if (b < d) {
      uint32_t s = b ? lower_bound_u32(N, k, prev) : 0u;  // inserted entries below entry b - 1
#pragma unroll
      for (uint32_t j = 0; j < 4; ++j) {
        const uint32_t i = b + j;
        if (i >= d) break;
        for (; s < k && N[s] < v[j]; ++s) out[i + s] = N[s];
        if (s) out[i + s] = v[j];
      }
      if (b + 4 >= d)
        for (; s < k; ++s) out[d + s] = N[s];
    }
  }
}

// Removes D (k >= 1 entries, sorted, all in L) from the sorted run L in
// place.  The tiles go from the bottom up: a tile is read before it is
// written, and writes nothing above its own entries.
template <uint32_t T>
__device__ void remove_run(uint32_t *L, uint32_t d, const uint32_t *D, uint32_t k, uint32_t t) {
  const uint32_t first = lower_bound_u32(L, d, D[0]) & ~3u;
  for (uint32_t base = first; base < d; base += 4 * T) {
    const uint32_t b = base + 4 * t;
    uint32_t v[4] = {0, 0, 0, 0};
    if (b < d) {
      const uint4 q = *reinterpret_cast<const uint4 *>(L + b);
      v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
    }
    sync_threads<T>();
    if (b < d) {
      uint32_t s = lower_bound_u32(D, k, v[0]);
#pragma unroll
      for (uint32_t j = 0; j < 4; ++j) {
        const uint32_t i = b + j;
        if (i >= d) break;
        while (s < k && D[s] < v[j]) ++s;
        if (s < k && D[s] == v[j]) continue;
        if (s) L[i - s] = v[j];
      }
    }
  }
}

// The slot offsets of x after k entries (sorted) joined or left its run: each
// moves by the entries of lower slots among them.
__device__ __forceinline__ void move_loff(const DevGraph &g, uint32_t x, const uint32_t *N, uint32_t k, bool joined,
                                          uint32_t t, uint32_t T) {
  uint32_t *lo = g.loff + (size_t)x * (g.nlt + 1);
  for (uint32_t s = t; s <= g.nlt; s += T) {
    const uint32_t m = s == g.nlt ? k : lower_bound_u32(N, k, s << kIdBits);
    lo[s] = joined ? lo[s] + m : lo[s] - m;
  }
}

// One source group's change, as the warp that selected it leaves it for the
// block when the run is long (k = 0: nothing for the block).
struct RunJob {
  uint32_t x, s, k, d, off, ncap;  // vertex, first selected entry, entries, degree, new run (units), its capacity (0: in place)
};

// Arena units (16 bytes) the insert may take: per source group, the run's
// new capacity when its degree plus every union insert of the group
// outgrows the capacity it has.
__global__ void k_arena_check(AdjUpdateArgs A) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  const uint32_t M = A.hdr->m, G = A.hdr->ngroups;
  if (blockIdx.x == 0 && threadIdx.x == 0) A.need16[1] = *A.g.arena_top;
  unsigned long long need = 0;
  for (uint32_t gi = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; gi < G; gi += warps) {
    const uint32_t s = A.dhead[gi], e = A.dhead[gi + 1];
    const uint32_t x = (uint32_t)(A.dkey[s] >> 32);
    uint32_t k = 0;
    for (uint32_t base = s; base < e; base += 32) {
      const uint32_t j = base + lane;
      bool sel = false;
      if (j < e) {
        const unsigned long long key = A.dkey[j];
        sel = (j == s || A.dkey[j - 1] != key) && (group_flag(A, M, x, (uint32_t)key & kIdMask) & 1u);
      }
      k += __popc(__ballot_sync(kFull, sel));
    }
    const uint32_t d = A.g.adj[x].y, c = A.g.cap[x];
    if (lane == 0 && d + k > c) {
      const uint32_t want = d + k;
      need += ((want + want / 4 + 4 + 3) & ~3u) / 4;
    }
  }
  if (lane == 0 && need) atomicAdd(&A.need16[0], need);
}

__global__ void __launch_bounds__(256) k_adj_insert(AdjUpdateArgs A) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t M = A.hdr->m, G = A.hdr->ngroups;
  // all or nothing: every warp takes the same decision from the values the
  // check left (the arena top as it was before this kernel)
  if (A.need16[1] + A.need16[0] > A.g.arena_words / 4) {
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(A.err, kErrArena);
    return;
  }
  __shared__ RunJob jobs[8];
  const uint32_t t = threadIdx.x, w = t >> 5;
  auto store = [&](const RunJob &J) {  // one thread, once the run is written
    if (J.ncap) {
      A.g.adj[J.x] = make_uint2(J.off, J.d + J.k);
      A.g.cap[J.x] = J.ncap;
      atomicAdd(A.relocations, 1ull);
    } else {
      A.g.adj[J.x].y = J.d + J.k;
    }
  };
  // neighbouring groups go to different blocks, so that a small batch's spread
  // over the SMs
  for (uint32_t g0 = 0; g0 < G; g0 += 8 * gridDim.x) {
    const uint32_t gi = g0 + w * gridDim.x + blockIdx.x;
    RunJob J{0, 0, 0, 0, 0, 0};
    const uint32_t *L = nullptr;
    if (gi < G) {
      const uint32_t s = A.dhead[gi], e = A.dhead[gi + 1];
      J.x = (uint32_t)(A.dkey[s] >> 32);
      J.s = s;
      const uint2 ax = A.g.adj[J.x];
      J.d = ax.y;
      J.off = ax.x;
      L = A.g.arena + (uint64_t)ax.x * 4;
      J.k = select_group(A, M, s, e, J.x, 1, true, L, J.d);
      const uint32_t need = J.d + J.k;
      if (J.k && need > A.g.cap[J.x]) {
        J.ncap = (need + need / 4 + 4 + 3) & ~3u;
        unsigned long long off16 = 0;
        if (lane == 0) off16 = atomicAdd(A.g.arena_top, (unsigned long long)(J.ncap / 4));
        off16 = __shfl_sync(kFull, off16, 0);
        if ((off16 + J.ncap / 4) * 4 > A.g.arena_words || off16 + J.ncap / 4 > 0xFFFFFFFFull) {
          if (lane == 0) atomicOr(A.err, kErrArena);
          J.k = 0;
        }
        J.off = (uint32_t)off16;
      }
      if (J.k && J.d < kLongRun) {
        const uint32_t *N = A.dsel + s;
        insert_run<32>(L, J.d, N, J.k, A.g.arena + (uint64_t)J.off * 4, lane);
        move_loff(A.g, J.x, N, J.k, true, lane, 32);
        if (lane == 0) store(J);
        J.k = 0;
      }
    }
    if (lane == 0) jobs[w] = J;
    if (!__syncthreads_or(J.k != 0)) continue;
    for (uint32_t j = 0; j < 8; ++j) {
      const RunJob B = jobs[j];
      if (B.k == 0) continue;
      const uint32_t *from = A.g.arena + (uint64_t)A.g.adj[B.x].x * 4, *N = A.dsel + B.s;
      insert_run<256>(from, B.d, N, B.k, A.g.arena + (uint64_t)B.off * 4, t);
      move_loff(A.g, B.x, N, B.k, true, t, 256);
      __syncthreads();  // every thread has read the old run's place
      if (t == 0) store(B);
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(256) k_adj_delete(AdjUpdateArgs A) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t M = A.hdr->m, G = A.hdr->ngroups;
  if (ld_volatile(*A.err) & kErrArena) return;  // the batch was refused: leave the graph as it was
  __shared__ RunJob jobs[8];
  const uint32_t t = threadIdx.x, w = t >> 5;
  for (uint32_t g0 = 0; g0 < G; g0 += 8 * gridDim.x) {
    const uint32_t gi = g0 + w * gridDim.x + blockIdx.x;
    RunJob J{0, 0, 0, 0, 0, 0};
    if (gi < G) {
      const uint32_t s = A.dhead[gi], e = A.dhead[gi + 1];
      J.x = (uint32_t)(A.dkey[s] >> 32);
      J.s = s;
      const uint2 ax = A.g.adj[J.x];
      J.d = ax.y;
      J.off = ax.x;
      uint32_t *L = A.g.arena + (uint64_t)ax.x * 4;
      J.k = select_group(A, M, s, e, J.x, 2, false, L, J.d);
      if (J.k && J.d < kLongRun) {
        const uint32_t *D = A.dsel + s;
        remove_run<32>(L, J.d, D, J.k, lane);
        move_loff(A.g, J.x, D, J.k, false, lane, 32);
        if (lane == 0) A.g.adj[J.x].y = J.d - J.k;
        J.k = 0;
      }
    }
    if (lane == 0) jobs[w] = J;
    if (!__syncthreads_or(J.k != 0)) continue;
    for (uint32_t j = 0; j < 8; ++j) {
      const RunJob B = jobs[j];
      if (B.k == 0) continue;
      const uint32_t *D = A.dsel + B.s;
      remove_run<256>(A.g.arena + (uint64_t)B.off * 4, B.d, D, B.k, t);
      move_loff(A.g, B.x, D, B.k, false, t, 256);
      if (t == 0) A.g.adj[B.x].y = B.d - B.k;
    }
    __syncthreads();
  }
}

__global__ void k_clear_touch(DevGraph g, const BatchHdr *hdr, const uint4 *upd, PackArgs P) {
  const uint32_t n = hdr->n;
  if (hdr->pack) {
    const size_t stride = (size_t)gridDim.x * blockDim.x, t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t *o32 = reinterpret_cast<uint32_t *>(P.out);
    unsigned long long *o64 = reinterpret_cast<unsigned long long *>(P.out + 64);
    for (size_t i = t; i < 16; i += stride) o32[i] = P.misc[i];
    for (size_t i = t; i < hdr->nseg; i += stride) o64[i] = P.segcnt[i];
    o32 = reinterpret_cast<uint32_t *>(o64 + hdr->nseg);
    for (size_t i = t; i < n; i += stride) o32[i] = P.vtp[i];
  }
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    uint4 u = upd[i];
    if (u.y < g.nv) atomicAnd(&g.lab[u.y], kLabelMask);
    if (u.z < g.nv) atomicAnd(&g.lab[u.z], kLabelMask);
  }
}

__global__ void k_arena_move(DevGraph g, const uint2 *nadj, uint32_t *narena) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < g.nv; v += warps) {
    const uint2 a = g.adj[v];
    const uint32_t *src = g.arena + (uint64_t)a.x * 4;
    uint32_t *dst = narena + (uint64_t)nadj[v].x * 4;
    for (uint32_t i = lane; i < a.y; i += 32) dst[i] = src[i];
  }
}

__global__ void k_edge_filter(DevGraph g) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < g.nv; v += warps) {
    const uint2 a = g.adj[v];
    const uint32_t *run = adj_list(g, a);
    for (uint32_t i = lane; i < a.y; i += 32) {
      const uint32_t w = run[i] & kIdMask;
      if (w < v) continue;  // each edge once
      uint32_t word;
      const uint32_t bits = bloom_bits(v, w, g.flt_mask, word);
      atomicOr(&g.flt[word], bits);
    }
  }
}

// Bound by the degrees' bytes; launched once per rebuild of the edge filter.
__global__ void k_entry_count(DevGraph g, unsigned long long *sum) {
  unsigned long long n = 0;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < g.nv; v += gridDim.x * blockDim.x) n += g.adj[v].y;
#pragma unroll
  for (uint32_t d = 16; d; d >>= 1) n += __shfl_xor_sync(kFull, n, d);
  if ((threadIdx.x & 31) == 0 && n) atomicAdd(sum, n);
}

__global__ void k_batch_clear(ClearArgs A) {
  const BatchHdr h = *reinterpret_cast<const BatchHdr *>(A.stage);
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t == 0) *A.hdr = h;
  auto copy = [&](void *to, unsigned long long from, size_t words) {
    const uint32_t *src = reinterpret_cast<const uint32_t *>(A.stage + from);
    for (size_t i = t; i < words; i += stride) static_cast<uint32_t *>(to)[i] = src[i];
  };
  copy(A.upd, h.o_up, 4ull * h.n);
  copy(A.bkey, h.o_bk, 2ull * h.m);
  copy(A.bidx, h.o_bi, h.m);
  copy(A.dkey, h.o_dk, 4ull * h.m);
  copy(A.dhead, h.o_dh, h.m ? h.ngroups + 1ull : 0ull);
  for (size_t i = t; i < A.job_ring; i += stride) A.job_seq[i] = i;
  for (size_t i = t; i < h.n; i += stride) A.vtp[i] = kNoView;
  for (size_t i = t; i < h.nseg; i += stride) A.segcnt[i] = 0;
  if (A.segwork)
    for (size_t i = t; i < h.nseg; i += stride) A.segwork[i] = 0;
  for (size_t i = t; i < h.nq_live; i += stride) A.qlisted[i] = 0;
  uint32_t *sc = reinterpret_cast<uint32_t *>(A.sc);
  for (size_t i = t; i < sizeof(Sched) / 4; i += stride) sc[i] = 0;
  for (size_t i = t; i < 64; i += stride) A.misc[i] = 0;
  for (size_t i = t; i <= h.bloom_mask; i += stride) A.bloom[i] = 0;
  for (size_t i = t; i <= h.bloom_mask >> 1; i += stride) A.table[i] = 0;
}

// ---------------------------------------------------------------------------
// Seeds (main.cu:268-329): update (a, b) x ordered query edge (u, v) with
// label(a) = label(u), label(b) = label(v) and, with a filter, a in C(u),
// b in C(v).
// ---------------------------------------------------------------------------
__global__ void k_seeds(SeedArgs A) {
  const uint32_t n = A.hdr->n;
  const unsigned long long seed_cap = A.hdr->seed_cap;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
  if (A.vtp[i] == kNoView) continue;
  uint4 u = A.upd[i];
  uint32_t a = u.y, b = u.z;
  // the engine validates updates on the host; callers that pass their own
  // device buffers (the allocation-free entry point) may not have: an id out
  // of range or a self loop seeds nothing
  if (a >= A.g.nv || b >= A.g.nv || a == b) continue;
  uint32_t la = A.g.lab[a] & kLabelMask, lb = A.g.lab[b] & kLabelMask;
  if (la >= 32 || lb >= 32) continue;
  uint32_t pb = la * 32 + lb;
  for (uint32_t e = A.pair_off[pb]; e < A.pair_off[pb + 1]; ++e) {
    uint32_t ent = A.pair_ent[e];
    if (A.only_slot != kAllSlots && (ent >> 8) != A.only_slot) continue;
    const QDev &q = A.qd[ent >> 8];
    if (q.bitmap) {
      const OrderRec &o = A.orders[q.order_base + (ent & 255)];
      uint32_t qa = o.vert[0], qb = o.vert[1];
      if (!((q.bitmap[(size_t)qa * q.col_len + (a >> 5)] >> (a & 31)) & 1u)) continue;
      if (!((q.bitmap[(size_t)qb * q.col_len + (b >> 5)] >> (b & 31)) & 1u)) continue;
    }
    unsigned long long s = atomicAdd(&A.sc->nseeds, 1ull);
    if (s < seed_cap) A.seeds[s] = make_uint4(i, ent, a, b);
  }
  }
  if (!A.arm) return;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&A.sc->armed, 1u) == gridDim.x - 1) {  // every block's seeds are counted
      unsigned long long total = ld_volatile(A.sc->nseeds);
      if (total > seed_cap) {
        A.sc->nseeds = total = seed_cap;
        atomicOr(&A.sc->error, kErrSeeds);
      }
      A.sc->outstanding.v = total + A.phantom;
      A.sc->done.v = total + A.phantom == 0 ? 1ull : 0ull;
    }
  }
}

}  // namespace

void launch_batch_clear(const ClearArgs &a, int blocks, cudaStream_t s) {
  k_batch_clear<<<blocks, 256, 0, s>>>(a);
}

void launch_edge_state(const EdgeStateArgs &a, int blocks, cudaStream_t s) {
  k_edge_state<<<blocks, 256, 0, s>>>(a);
}

void launch_arena_check(const AdjUpdateArgs &a, int blocks, cudaStream_t s) {
  k_arena_check<<<blocks, 256, 0, s>>>(a);
}

void launch_arena_move(DevGraph g, const uint2 *nadj, uint32_t *narena, int blocks, cudaStream_t s) {
  k_arena_move<<<blocks, 256, 0, s>>>(g, nadj, narena);
}

void launch_edge_filter(DevGraph g, int blocks, cudaStream_t s) { k_edge_filter<<<blocks, 256, 0, s>>>(g); }

void launch_entry_count(DevGraph g, unsigned long long *sum, int blocks, cudaStream_t s) {
  k_entry_count<<<blocks, 256, 0, s>>>(g, sum);
}

void launch_adj_insert(const AdjUpdateArgs &a, int blocks, cudaStream_t s) {
  k_adj_insert<<<blocks, 256, 0, s>>>(a);
}

void launch_adj_delete(const AdjUpdateArgs &a, int blocks, cudaStream_t s) {
  k_adj_delete<<<blocks, 256, 0, s>>>(a);
}

void launch_clear_touch(DevGraph g, const BatchHdr *hdr, const uint4 *upd, const PackArgs &p, int blocks,
                        cudaStream_t s) {
  k_clear_touch<<<blocks, 256, 0, s>>>(g, hdr, upd, p);
}

void launch_seeds(const SeedArgs &a, int blocks, cudaStream_t s) {
  k_seeds<<<blocks, 256, 0, s>>>(a);
}

}  // namespace dsm
