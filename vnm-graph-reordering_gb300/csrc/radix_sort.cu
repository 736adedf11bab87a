// Stable LSD radix sort of 64-bit keys with a 32-bit payload.
//
// Used wherever the path needs an order the reference gets from std::sort or
// Python's sorted(): the (row, col) order of a COO (customSort,
// mtx/readMtx.hpp:56-82), the VNM row order (reordering.py:219) and the
// compressor's (block, segment) grouping.  Keys are unique or ties are
// broken by the payload's original position, so stability makes the result
// identical to the reference's.
//
// One pass per 8-bit digit: (1) per-tile digit histograms, (2) the place of
// every (digit, tile), (3) a stable scatter in which every warp ranks its
// contiguous chunk of the tile by votes, once, the keys and
// their ranks staying in registers until the chunk's place is known.  Up to
// RS_DIRECT tiles the scatter itself adds up the histograms of the tiles
// before its own (step 2 as two launches of a prefix sum cost more than those
// reads); longer arrays scan (digit, tile) in digit-major order.  Bound by
// latency up to a few 100 K keys: a pass over 228 K keys took 24 us with the
// keys read and ranked twice and a separate scan, 13 us now.
// Only the low `bits` bits of the keys are sorted on, so callers pack keys
// tightly to save passes.
#include "common.cuh"

namespace vnm {

// Lanes of a converged warp with this lane's digit (`ok` lanes only), by one
// vote a bit: a pass over 228 K keys took 9.8 us with it, 10.8 with
// __match_any_sync.
__device__ __forceinline__ unsigned warp_peers(unsigned d, bool ok) {
  unsigned peers = __ballot_sync(0xffffffffu, ok);
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const bool on = (d >> b) & 1u;
    const unsigned v = __ballot_sync(0xffffffffu, on);
    peers &= on ? v : ~v;
  }
  return peers;
}


constexpr int RS_NT = 512;           // threads per tile
constexpr int RS_PER = 8;            // keys per thread
constexpr int RS_TILE = RS_NT * RS_PER;
constexpr int RS_WARPS = RS_NT / 32;
constexpr int RS_CHUNK = RS_TILE / RS_WARPS;  // keys per warp, in order
constexpr int RS_DIRECT = 128;       // tiles

// direct: hist[tile][digit] and the digits' totals added to tot; else hist[digit][tile].
__global__ void __launch_bounds__(RS_NT) k_rs_hist(const unsigned long long* keys, int n, int shift, int* hist,
                                                    int ntiles, int* tot) {
  __shared__ int h[256];
  const int base = blockIdx.x * RS_TILE + threadIdx.x;
  unsigned d[RS_PER];
#pragma unroll
  for (int q = 0; q < RS_PER; ++q)
    d[q] = base + q * RS_NT < n ? (unsigned)(keys[base + q * RS_NT] >> shift) & 255u : 256u;
  if (threadIdx.x < 256) h[threadIdx.x] = 0;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < RS_PER; ++q)
    if (d[q] < 256u) atomicAdd(&h[d[q]], 1);
  __syncthreads();
  if (threadIdx.x < 256) {
    const int c = h[threadIdx.x];
    if (tot) {
      hist[blockIdx.x * 256 + threadIdx.x] = c;
      if (c) atomicAdd(&tot[threadIdx.x], c);
    } else {
      hist[threadIdx.x * ntiles + blockIdx.x] = c;
    }
  }
}

// offs: the scanned hist[digit][tile], or (tot given) the hist[tile][digit] of k_rs_hist.
__global__ void __launch_bounds__(RS_NT) k_rs_scatter(const unsigned long long* keys, const int* vals, int n,
                                                       int shift, const int* offs, int ntiles, const int* tot,
                                                       unsigned long long* okeys, int* ovals) {
  __shared__ int wcount[RS_WARPS][256];  // per warp, per digit: keys in the warp's chunk, then before it
  __shared__ int part[2][256];
  __shared__ int wsum[8];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int base = blockIdx.x * RS_TILE + w * RS_CHUNK + lane;
  unsigned long long k[RS_PER];
  int v[RS_PER];
#pragma unroll
  for (int q = 0; q < RS_PER; ++q) {
    const int i = base + 32 * q;
    k[q] = i < n ? keys[i] : 0ull;
    v[q] = i >= n ? 0 : vals ? vals[i] : i;
  }
  int before = 0;  // this digit's keys in earlier tiles (direct: every other one of them)
  const int dg = tid & 255, half = tid >> 8;
  if (tot) {
#pragma unroll 8
    for (int t = half; t < (int)blockIdx.x; t += 2) before += offs[t * 256 + dg];
  } else if (half == 0) {
    before = offs[dg * ntiles + blockIdx.x];
  }
  for (int d = lane; d < 256; d += 32) wcount[w][d] = 0;
  __syncwarp();
  unsigned short rank[RS_PER];
#pragma unroll
  for (int q = 0; q < RS_PER; ++q) {
    const bool ok = base + 32 * q < n;
    const unsigned d = (unsigned)(k[q] >> shift) & 255u;
    const unsigned peers = warp_peers(d, ok);
    rank[q] = ok ? (unsigned short)(wcount[w][d] + __popc(peers & ((1u << lane) - 1u))) : 0;
    __syncwarp();
    if (ok && lane == __ffs(peers) - 1) wcount[w][d] += __popc(peers);
    __syncwarp();
  }
  part[half][dg] = before;
  int incl = 0, mine = 0;
  if (tot && tid < 256) {  // the digit's start: the totals of the digits before it
    incl = mine = tot[tid];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) wsum[w] = incl;
  }
  __syncthreads();
  if (tid < 256) {  // where each warp's keys of the digit go
    int run = part[0][tid];
    if (tot) {
      run += part[1][tid] + incl - mine;
      for (int u = 0; u < w; ++u) run += wsum[u];
    }
#pragma unroll
    for (int u = 0; u < RS_WARPS; ++u) {
      const int c = wcount[u][tid];
      wcount[u][tid] = run;
      run += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < RS_PER; ++q)
    if (base + 32 * q < n) {
      const int dst = wcount[w][(unsigned)(k[q] >> shift) & 255u] + rank[q];
      okeys[dst] = k[q];
      ovals[dst] = v[q];
    }
}

size_t radix_sort_scratch_bytes(int n) {
  const int ntiles = (n + RS_TILE - 1) / RS_TILE;
  size_t b = 2 * arena_bytes(n, sizeof(unsigned long long)) + 2 * arena_bytes(n, sizeof(int));
  b += 2 * arena_bytes((size_t)256 * ntiles, sizeof(int)) + arena_bytes(8 * 256, sizeof(int));
  b += 8 * scan_scratch_bytes(256 * ntiles);
  return b + 4096;
}

// Sort keys[0..n) ascending, carrying vals (nullptr = original positions).
// Results land in *out_keys / *out_vals (arena memory or the inputs).
// `bits` = number of low key bits that can be nonzero (<= 64).
vnm_status radix_sort_u64(vnm_ctx* ctx, const unsigned long long* keys, const int* vals, int n, int bits,
                          unsigned long long** out_keys, int** out_vals) {
  if (n <= 0) {
    *out_keys = const_cast<unsigned long long*>(keys);
    *out_vals = const_cast<int*>(vals);
    return VNM_OK;
  }
  const int ntiles = (n + RS_TILE - 1) / RS_TILE;
  const bool direct = ntiles <= RS_DIRECT;
  unsigned long long* kb[2] = {arena_take<unsigned long long>(ctx, n), arena_take<unsigned long long>(ctx, n)};
  int* vb[2] = {arena_take<int>(ctx, n), arena_take<int>(ctx, n)};
  int* hist = arena_take<int>(ctx, (size_t)256 * ntiles);
  int* offs = arena_take<int>(ctx, (size_t)256 * ntiles);
  int* tot = arena_take<int>(ctx, 8 * 256);
  if (!kb[0] || !kb[1] || !vb[0] || !vb[1] || !hist || !offs || !tot) return VNM_ERR_NOMEM;
  if (direct) VNM_CUDA_TRY(cudaMemsetAsync(tot, 0, sizeof(int) * 8 * 256, ctx->stream));
  const unsigned long long* ck = keys;
  const int* cv = vals;
  int cur = 0;
  for (int shift = 0; shift < bits; shift += 8) {
    int* t = direct ? tot + 256 * (shift / 8) : nullptr;
    VNM_LAUNCH(ctx, k_rs_hist, ntiles, RS_NT, 0, ck, n, shift, hist, ntiles, t);
    if (!direct) VNM_TRY(exclusive_scan(ctx, hist, offs, 256 * ntiles, nullptr));
    VNM_LAUNCH(ctx, k_rs_scatter, ntiles, RS_NT, 0, ck, cv, n, shift, direct ? hist : offs, ntiles, t, kb[cur], vb[cur]);
    ck = kb[cur];
    cv = vb[cur];
    cur ^= 1;
  }
  *out_keys = const_cast<unsigned long long*>(ck);
  *out_vals = const_cast<int*>(cv);
  return VNM_OK;
}

}  // namespace vnm
