// Listed results on the device: the matcher's table (segment, tuple rows in
// whatever order warps found them) becomes each (query, update) segment's
// tuples, back to back and in canonical order, before anything crosses to
// the host.  No reference counterpart (it emits no embeddings).
//
//   k_list_sum, k_list_offsets   where each segment's tuples go: a scan of the
//                                counts that are listed (not over the work
//                                limit, the query within its listing budget)
//   k_list_place                 rows to their segments (a cursor per segment)
//   k_list_sort_small            segments of 2..32 tuples, a warp each
//   k_list_sort_chunks           longer ones, 1024 tuples at a time, in shared memory
//   k_list_merge                 those runs merged pairwise, a launch per doubling
//
// The first two belong to the batch's first segment (their sizes come from
// the batch header); the others are launched once the host knows the totals.
// Before, the raw table crossed to the host, with every partial tuple of the
// searches that went over their limit, and was scattered and sorted on host
// threads.  A burst of nine requests against 64 queries (0.8 million tuples
// listed, 5,300 searches over their limit): device time of a merged batch with
// its download 18.5 -> 6.5 ms, the burst 120 -> 45 ms.  One batch of 305,000
// tuples of 5: placed in 14 us and sorted in 165 us, where the host took 2.1 ms
// to sort; the call 7.2 -> 2.1 ms.
#include <algorithm>

#include "kernels.cuh"

namespace dsm {

namespace {

constexpr uint32_t kChunk = 1024;  // tuples sorted together in shared memory (16 words: 70 KB of it)
constexpr uint32_t kSmall = 32;    // a warp sorts these by rank, without shared indices or barriers

// Tuples of segment s that are listed.
__device__ __forceinline__ unsigned long long listed(const ListArgs &A, uint32_t n, unsigned long long s) {
  const unsigned long long c = A.segcnt[s];
  if (c == 0 || (c & kCountIncomplete)) return 0;
  return A.qlimit && A.qlisted[s / n] > A.qlimit ? 0 : c;
}
__device__ __forceinline__ unsigned long long chunks_of(unsigned long long c) {
  return c > kSmall ? (c + kChunk - 1) / kChunk : 0;
}

struct Totals {
  unsigned long long words, chunks, most;
};

// Sum (and maximum) over a block of 256 threads, in every thread.
__device__ Totals block_total(Totals v) {
  __shared__ Totals part[8];
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (uint32_t d = 16; d; d >>= 1) {
    v.words += __shfl_xor_sync(kFull, v.words, d);
    v.chunks += __shfl_xor_sync(kFull, v.chunks, d);
    v.most = max(v.most, __shfl_xor_sync(kFull, v.most, d));
  }
  __syncthreads();  // the last call's parts have been read
  if (lane == 0) part[w] = v;
  __syncthreads();
  Totals t = part[0];
  for (uint32_t k = 1; k < 8; ++k) {
    t.words += part[k].words;
    t.chunks += part[k].chunks;
    t.most = max(t.most, part[k].most);
  }
  return t;
}

__device__ __forceinline__ unsigned long long per_block(unsigned long long nseg) {
  return (nseg + gridDim.x - 1) / gridDim.x;
}

__global__ void __launch_bounds__(256) k_list_sum(ListArgs A) {
  const unsigned long long nseg = A.hdr->nseg, per = per_block(nseg);
  const uint32_t n = A.hdr->n;
  const unsigned long long lo = min(blockIdx.x * per, nseg), hi = min(lo + per, nseg);
  Totals v{0, 0, 0};
  for (unsigned long long s = lo + threadIdx.x; s < hi; s += 256) {
    const unsigned long long c = listed(A, n, s);
    v.words += c * A.widths[s / n];
    v.chunks += chunks_of(c);
    v.most = max(v.most, c);
  }
  v = block_total(v);
  if (threadIdx.x == 0) {
    A.partial[3 * blockIdx.x] = v.words;
    A.partial[3 * blockIdx.x + 1] = v.chunks;
    A.partial[3 * blockIdx.x + 2] = v.most;
  }
}

// kAlone: one block for all segments, which sums them itself.
template <bool kAlone>
__global__ void __launch_bounds__(256) k_list_offsets(ListArgs A) {
  __shared__ unsigned long long s_words[8];
  __shared__ uint32_t s_chunks[8];
  const unsigned long long nseg = A.hdr->nseg, per = per_block(nseg);
  const uint32_t n = A.hdr->n, t = threadIdx.x, lane = t & 31, w = t >> 5;
  const unsigned long long lo = min(blockIdx.x * per, nseg), hi = min(lo + per, nseg);
  // the blocks before this one (the grid is kListBlocks = 256 blocks)
  Totals before{0, 0, 0}, all{0, 0, 0};
  if constexpr (kAlone) {
    for (unsigned long long s = t; s < nseg; s += 256) {
      const unsigned long long c = listed(A, n, s);
      all.words += c * A.widths[s / n];
      all.chunks += chunks_of(c);
      all.most = max(all.most, c);
    }
  } else if (t < gridDim.x) {
    all = Totals{A.partial[3 * t], A.partial[3 * t + 1], A.partial[3 * t + 2]};
    if (t < blockIdx.x) before = all;
  }
  before = block_total(before);
  all = block_total(all);
  if (blockIdx.x == 0 && t == 0) {
    A.totals[0] = all.words;
    A.totals[1] = all.chunks;
    A.totals[2] = all.most;
    A.off[nseg] = all.words;
    A.chunk[nseg] = (uint32_t)all.chunks;
  }
  unsigned long long words = before.words;
  uint32_t chunks = (uint32_t)before.chunks;
  for (unsigned long long base = lo; base < hi; base += 256) {
    const unsigned long long s = base + t;
    const unsigned long long c = s < hi ? listed(A, n, s) : 0, x = s < hi ? c * A.widths[s / n] : 0;
    const uint32_t y = (uint32_t)chunks_of(c);
    unsigned long long ix = x;
    uint32_t iy = y;
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
      const unsigned long long px = __shfl_up_sync(kFull, ix, d);
      const uint32_t py = __shfl_up_sync(kFull, iy, d);
      if (lane >= d) {
        ix += px;
        iy += py;
      }
    }
    __syncthreads();  // the last round's sums have been read
    if (lane == 31) {
      s_words[w] = ix;
      s_chunks[w] = iy;
    }
    __syncthreads();
    unsigned long long bx = 0, tx = 0;
    uint32_t by = 0, ty = 0;
    for (uint32_t k = 0; k < 8; ++k) {
      if (k < w) {
        bx += s_words[k];
        by += s_chunks[k];
      }
      tx += s_words[k];
      ty += s_chunks[k];
    }
    if (s < hi) {
      A.off[s] = words + bx + ix - x;
      A.chunk[s] = chunks + by + iy - y;
      A.cursor[s] = 0;
    }
    words += tx;
    chunks += ty;
  }
}

// Bound by the rows' bytes.  The rows one warp emitted together share their
// segment, so a warp's rows of one segment take their places with one addition.
__global__ void k_list_place(ListArgs A, const uint32_t *seg, const uint32_t *rows, uint32_t W,
                             unsigned long long cnt, uint32_t *out) {
  const uint32_t n = A.hdr->n, lane = threadIdx.x & 31;
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long r = blockIdx.x * blockDim.x + threadIdx.x; r - lane < cnt; r += stride) {
    const uint32_t s = r < cnt ? seg[r] : 0xFFFFFFFFu;
    unsigned long long o = 0, e = 0;
    if (r < cnt) {
      o = A.off[s];
      e = A.off[s + 1];
    }
    const bool keep = e > o;  // a listed segment (rows of the others are left behind)
    const uint32_t peers = __match_any_sync(kFull, keep ? s : 0xFFFFFFFFu);
    uint32_t p = 0;
    const uint32_t leader = __ffs(peers) - 1;
    if (keep && lane == leader) p = atomicAdd(&A.cursor[s], (uint32_t)__popc(peers));
    p = __shfl_sync(kFull, p, leader) + __popc(peers & lanemask_lt());
    if (!keep) continue;
    const uint32_t w = A.widths[s / n];
    const uint32_t *src = rows + r * W;
    uint32_t *dst = out + o + (unsigned long long)p * w;
    for (uint32_t k = 0; k < w; ++k) dst[k] = src[k];
  }
}

__device__ __forceinline__ bool row_less(const uint32_t *a, const uint32_t *b, uint32_t w) {
  for (uint32_t k = 0; k < w; ++k)
    if (a[k] != b[k]) return a[k] < b[k];
  return false;
}

// Segments of 2..32 tuples: a warp holds one in shared memory, each lane
// counts the tuples below its own and writes it there.
__global__ void __launch_bounds__(256) k_list_sort_small(ListArgs A, uint32_t *out) {
  __shared__ uint32_t s_rows[8][kSmall * 17];
  const uint32_t n = A.hdr->n, lane = threadIdx.x & 31;
  const unsigned long long nseg = A.hdr->nseg, warps = (unsigned long long)gridDim.x * 8;
  uint32_t *R = s_rows[threadIdx.x >> 5];
  for (unsigned long long base = (blockIdx.x * 8ull + (threadIdx.x >> 5)) * 32; base < nseg; base += warps * 32) {
    const unsigned long long s = base + lane;
    unsigned long long o = 0;
    uint32_t w = 1, c = 0;
    if (s < nseg) {
      o = A.off[s];
      w = A.widths[s / n];
      c = (uint32_t)min((A.off[s + 1] - o) / w, (unsigned long long)kSmall + 1);
    }
    for (uint32_t m = __ballot_sync(kFull, c >= 2 && c <= kSmall); m; m &= m - 1) {
      const uint32_t k = __ffs(m) - 1;
      const uint32_t ck = __shfl_sync(kFull, c, k), wk = __shfl_sync(kFull, w, k), st = wk | 1;
      uint32_t *seg = out + __shfl_sync(kFull, o, k);
      for (uint32_t e = lane; e < ck * wk; e += 32) R[e / wk * st + e % wk] = seg[e];
      __syncwarp();
      if (lane < ck) {
        const uint32_t *mine = R + lane * st;
        uint32_t rank = 0;
        for (uint32_t j = 0; j < ck; ++j) rank += row_less(R + j * st, mine, wk);
        for (uint32_t j = 0; j < wk; ++j) seg[rank * wk + j] = mine[j];
      }
      __syncwarp();
    }
  }
}

// The segment of chunk b: the last one whose first chunk is at or before it
// (segments without chunks share the next one's first chunk).
__device__ __forceinline__ unsigned long long segment_of(const uint32_t *chunk, unsigned long long nseg, uint32_t b) {
  unsigned long long lo = 0, hi = nseg;
  while (lo + 1 < hi) {
    const unsigned long long mid = (lo + hi) >> 1;
    if (chunk[mid] <= b) lo = mid; else hi = mid;
  }
  return lo;
}

// One block per chunk of up to 1024 tuples: the rows in shared memory (an odd
// stride, so that equal columns fall into different banks), a bitonic sort of
// their 16-bit indices, the rows written out in order.  A segment of one chunk
// ends in `out`; the runs of longer ones go to `runs`, where the merges start.
__global__ void __launch_bounds__(256) k_list_sort_chunks(ListArgs A, uint32_t *out, uint32_t *runs) {
  extern __shared__ uint32_t sm[];
  __shared__ unsigned long long s_seg;
  const uint32_t t = threadIdx.x, n = A.hdr->n;
  if (t == 0) s_seg = segment_of(A.chunk, A.hdr->nseg, blockIdx.x);
  __syncthreads();
  const unsigned long long s = s_seg, o = A.off[s];
  const uint32_t w = A.widths[s / n], st = w | 1;
  const unsigned long long c = (A.off[s + 1] - o) / w, r0 = (unsigned long long)(blockIdx.x - A.chunk[s]) * kChunk;
  const uint32_t rows = (uint32_t)min((unsigned long long)kChunk, c - r0);
  uint16_t *idx = reinterpret_cast<uint16_t *>(sm);  // first, then the rows
  uint32_t *R = sm + kChunk / 2;
  const uint32_t *src = out + o + r0 * w;
  for (uint32_t e = t; e < rows * w; e += 256) R[e / w * st + e % w] = src[e];
  uint32_t P = 64;
  while (P < rows) P <<= 1;
  for (uint32_t i = t; i < P; i += 256) idx[i] = i < rows ? (uint16_t)i : 0xFFFFu;
  __syncthreads();
  for (uint32_t k = 2; k <= P; k <<= 1)
    for (uint32_t j = k >> 1; j; j >>= 1) {
      for (uint32_t i = t; i < P / 2; i += 256) {
        const uint32_t a = 2 * i - (i & (j - 1)), b = a + j;
        const uint32_t ia = idx[a], ib = idx[b];
        // absent rows come last
        const bool gt = ib == 0xFFFFu ? false : ia == 0xFFFFu ? true : row_less(R + ib * st, R + ia * st, w);
        const bool lt = ia == 0xFFFFu ? false : ib == 0xFFFFu ? true : !gt;
        if ((a & k) == 0 ? gt : lt) {
          idx[a] = (uint16_t)ib;
          idx[b] = (uint16_t)ia;
        }
      }
      __syncthreads();
    }
  uint32_t *dst = (c > kChunk ? runs : out) + o + r0 * w;
  for (uint32_t e = t; e < rows * w; e += 256) dst[e] = R[idx[e / w] * st + e % w];
}

// Merges the sorted runs of `run` tuples pairwise: each tuple's place is its
// place in its own run plus the tuples below it in the other (tuples of a
// segment differ).  A run without a partner is copied.
__global__ void __launch_bounds__(256) k_list_merge(ListArgs A, const uint32_t *src, uint32_t *dst,
                                                    unsigned long long run) {
  __shared__ unsigned long long s_seg;
  const uint32_t t = threadIdx.x, n = A.hdr->n;
  if (t == 0) s_seg = segment_of(A.chunk, A.hdr->nseg, blockIdx.x);
  __syncthreads();
  const unsigned long long s = s_seg, o = A.off[s];
  const uint32_t w = A.widths[s / n];
  const unsigned long long c = (A.off[s + 1] - o) / w, r0 = (unsigned long long)(blockIdx.x - A.chunk[s]) * kChunk;
  if (c <= kChunk) return;
  const uint32_t *base = src + o;
  for (unsigned long long i = r0 + t; i < min(r0 + kChunk, c); i += 256) {
    const unsigned long long mine = i / run * run, pair = i / (2 * run) * (2 * run);
    const unsigned long long other = mine == pair ? min(pair + run, c) : pair, end = min(other + run, c);
    const uint32_t *x = base + i * w;
    unsigned long long lo = other, hi = end;
    while (lo < hi) {
      const unsigned long long mid = (lo + hi) >> 1;
      if (row_less(base + mid * w, x, w)) lo = mid + 1; else hi = mid;
    }
    uint32_t *to = dst + o + (pair + (i - mine) + (lo - other)) * w;
    for (uint32_t k = 0; k < w; ++k) to[k] = x[k];
  }
}

// Shared memory of a sort block for tuples of up to W words.
constexpr int sort_smem(uint32_t W) { return (int)(kChunk * 2 + kChunk * (W | 1) * 4); }

}  // namespace

cudaError_t list_prepare() {
  return cudaFuncSetAttribute(k_list_sort_chunks, cudaFuncAttributeMaxDynamicSharedMemorySize, sort_smem(kMaxWidth));
}

int launch_list_scan(const ListArgs &a, size_t nseg, cudaStream_t s) {
  if (nseg && nseg <= 2048) {  // eight rounds of one block: no longer than the launch it saves (4 us)
    k_list_offsets<true><<<1, 256, 0, s>>>(a);
    return 1;
  }
  k_list_sum<<<kListBlocks, 256, 0, s>>>(a);
  k_list_offsets<false><<<kListBlocks, 256, 0, s>>>(a);
  return 2;
}

void launch_list_place(const ListArgs &a, const uint32_t *seg, const uint32_t *rows, uint32_t W,
                       unsigned long long cnt, uint32_t *out, int num_sms, cudaStream_t s) {
  const unsigned blocks = (unsigned)std::min<unsigned long long>((cnt + 255) / 256, num_sms * 8ull);
  k_list_place<<<std::max(blocks, 1u), 256, 0, s>>>(a, seg, rows, W, cnt, out);
}

int launch_list_sort(const ListArgs &a, uint32_t W, unsigned long long nseg, unsigned long long chunks,
                     unsigned long long most, uint32_t *out, uint32_t *scratch, int num_sms, cudaStream_t s) {
  const unsigned blocks = (unsigned)std::min<unsigned long long>((nseg + 255) / 256, num_sms * 4ull);
  k_list_sort_small<<<std::max(blocks, 1u), 256, 0, s>>>(a, out);
  int launched = 1;
  if (!chunks) return launched;
  int passes = 0;
  for (unsigned long long run = kChunk; run < most; run *= 2) ++passes;
  // the last pass ends in `out`
  k_list_sort_chunks<<<(unsigned)chunks, 256, sort_smem(W), s>>>(a, out, passes & 1 ? scratch : out);
  ++launched;
  uint32_t *src = passes & 1 ? scratch : out, *dst = passes & 1 ? out : scratch;
  unsigned long long run = kChunk;
  for (int p = 0; p < passes; ++p, run *= 2) {
    k_list_merge<<<(unsigned)chunks, 256, 0, s>>>(a, src, dst, run);
    std::swap(src, dst);
    ++launched;
  }
  return launched;
}

}  // namespace dsm
