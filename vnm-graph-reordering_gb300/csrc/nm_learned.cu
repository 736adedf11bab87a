// Learned-proposal reorder: a parallel, conflict-free swap-matching search
// whose candidate swaps are ranked by a small MLP before exact scoring.
//
// The reference's greedy (reorder/reorder.h:1805-2474) visits at most M+1
// segments per round and scores every one of their M*M swaps exactly; it is
// sequential by construction.  This mode is a different search with the same
// objective (fewer invalid M-groups, i.e. more retained nonzeros) built for a
// GPU: every round, every invalid segment p proposes swaps with the nodes of
// KT sampled target segments, the MLP scores all of them, only the best 8 per
// segment are scored exactly (the integer kernel decides), and a claim-based
// matching accepts at most one improving swap per segment, so the accepted
// swaps touch disjoint segments and their exact gains add up.  An exhaustive
// mode scores every candidate exactly instead (the fallback and the baseline
// the network is measured against).
//
// State in HBM, all indexed by original ids (rows never move; only which node
// sits at which column position does):
//   G[r * nseg + s]  the M-bit group of row r in segment s (bit i = the column
//                    at position s*M+i), R * nseg bytes;
//   cnt[s]           rows whose group in s has more than N bits;
//   hist[s][k]       rows whose group in s has exactly k bits (k = 0..8);
//   colh[u][k]       rows of column u whose group (in u's segment) has k bits.
//
// MLP: 32 features -> 128 -> 128 -> 1 (ReLU), BF16 operands, FP32
// accumulation.  Inference runs on tcgen05: a CTA builds the features of
// 128 candidates into shared memory, two chained MMAs go through tensor
// memory, and the last layer is a dot product in registers.
#include <cuda_bf16.h>

#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "sm100_ptx.cuh"

namespace vnm {

constexpr int LF = 32;       // features
constexpr int LH = 128;      // hidden width
constexpr int LTOP = 8;      // proposals per segment that are scored exactly
constexpr uint32_t L_WAIT = 1u << 22;

struct LMat {  // one matrix's state
  int R, M, N, nseg;
  int obj;    // 0: invalid groups, 1: retained nonzeros
  const int* cptr;
  const int* crow;
  int* orig;  // position -> node
  int* pos;   // node -> position
  unsigned char* G;
  int* cnt;
  int* hist;  // [nseg * 9]
  int* colh;  // [R * 9]
};

// ---------------------------------------------------------------------------
// State build and maintenance
// ---------------------------------------------------------------------------
__global__ void k_l_build_G(const int* row, const int* col, const float* val, int nnz, int M, int nseg, unsigned* Gw) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nnz; i += gridDim.x * blockDim.x) {
    if (val[i] == 0.0f) continue;
    const long long cell = (long long)row[i] * nseg + col[i] / M;
    atomicOr(&Gw[cell >> 2], (1u << (col[i] % M)) << ((cell & 3) * 8));
  }
}

// hist / cnt of a segment from its columns' histograms: a group of k bits is
// counted by each of its k columns.  (Counting runs of the sorted pattern with
// atomics took 44 us at 65536 rows, 2 M entries; this takes 7.)
__global__ void k_l_seg_hist(LMat L) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < L.nseg; s += gridDim.x * blockDim.x) {
    int h[9], t = 0, c = 0;
#pragma unroll
    for (int k = 1; k <= 8; ++k) h[k] = 0;
    for (int i = 0; i < L.M; ++i) {
      const int u = L.orig[s * L.M + i];
#pragma unroll
      for (int k = 1; k <= 8; ++k) h[k] += L.colh[u * 9 + k];
    }
#pragma unroll
    for (int k = 1; k <= 8; ++k) {
      h[k] /= k;
      L.hist[s * 9 + k] = h[k];
      t += h[k];
      c += k > L.N ? h[k] : 0;
    }
    L.hist[s * 9] = L.R - t;
    L.cnt[s] = c;
  }
}

// colh of the columns at some positions.  A column's rows are cut into chunks
// of L_CHUNK, one warp a chunk, so a hub column spreads over many warps.
// take_column zeroes a column's histogram and appends its chunks to the work
// list, k_l_colh_rows adds each chunk's histogram.  (The sums are of
// integers, so the list's order does not matter, and it is made by one atomic
// a warp; with chunk counts, a scan of them over all R columns and a search
// in the offsets for each chunk, a round of the search took five launches
// and 25 us more at 65536 rows.)
constexpr int L_CHUNK = 256;
constexpr int L_ROWS = L_CHUNK / 32;  // a lane's rows of a chunk, all in flight (one after the other,
                                      // k_l_colh_rows took 195 us of eleven rounds and k_l_apply_rows 180, 152 and 142 now)

// Counters of a call, on the device.
enum { LC_ACTIVE, LC_ACC, LC_SWAP_ITEMS, LC_DUMP, LC_ERR, LC_COL_ITEMS, LC_N = 8 };

__device__ __forceinline__ int chunks_of(const LMat& L, int u) {
  return (L.cptr[u + 1] - L.cptr[u] + L_CHUNK - 1) / L_CHUNK;
}

// Where a lane's n items go in a list of *len: whole warps call.
__device__ __forceinline__ int warp_append(int n, int* len) {
  const int lane = threadIdx.x & 31;
  int incl = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  int base = 0;
  if (lane == 31 && incl > 0) base = atomicAdd(len, incl);
  return __shfl_sync(0xffffffffu, base, 31) + incl - n;
}

// items: (position, chunk); whole warps call, lanes without a column with live = false
__device__ __forceinline__ void take_column(const LMat& L, int a, bool live, int2* items, int* nitems) {
  int c = 0;
  if (live) {
    const int u = L.orig[a];
#pragma unroll
    for (int z = 0; z < 9; ++z) L.colh[u * 9 + z] = 0;
    c = chunks_of(L, u);
  }
  const int at = warp_append(c, nitems);
  for (int k = 0; k < c; ++k) items[at + k] = make_int2(a, k);
}

__global__ void k_l_all_columns(LMat L, int2* items, int* nitems) {
  const int lane = threadIdx.x & 31;
  for (int a0 = blockIdx.x * blockDim.x + threadIdx.x - lane; a0 < L.R; a0 += gridDim.x * blockDim.x)
    take_column(L, a0 + lane, a0 + lane < L.R, items, nitems);
}

__global__ void k_l_colh_rows(LMat L, const int2* items, const int* nitems) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  const int tot = *nitems;
  for (int item = warp; item < tot; item += nw) {
    const int2 it = items[item];
    const int u = L.orig[it.x], s = it.x / L.M;
    const int beg = L.cptr[u] + it.y * L_CHUNK;
    const int end = min(beg + L_CHUNK, L.cptr[u + 1]);
    int r[L_ROWS], k[L_ROWS], h[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int x = 0; x < L_ROWS; ++x) r[x] = beg + lane + 32 * x < end ? L.crow[beg + lane + 32 * x] : -1;
#pragma unroll
    for (int x = 0; x < L_ROWS; ++x) k[x] = r[x] >= 0 ? __popc(L.G[(long long)r[x] * L.nseg + s]) : -1;
#pragma unroll
    for (int x = 0; x < L_ROWS; ++x)
#pragma unroll
      for (int z = 0; z < 9; ++z) h[z] += (k[x] == z);
#pragma unroll
    for (int z = 0; z < 9; ++z) {
      const int v = __reduce_add_sync(0xffffffffu, h[z]);
      if (lane == z && v) atomicAdd(&L.colh[u * 9 + z], v);
    }
  }
}

// The round's start: the segments that hold an invalid group in ascending
// order to `active` (block 0, a tile of its threads x 4 at a time: 8192
// segments are two tiles), the round's counters and the best and claim words
// cleared (the other blocks).  One launch where a scan took four and 18 us.
constexpr int L_START_THREADS = 1024;
__global__ void __launch_bounds__(L_START_THREADS)
    k_l_round_start(LMat L, int* active, int* ci, unsigned long long* best, unsigned long long* claim) {
  if (blockIdx.x > 0) {
    for (int s = (blockIdx.x - 1) * blockDim.x + threadIdx.x; s < L.nseg; s += (gridDim.x - 1) * blockDim.x)
      best[s] = claim[s] = 0ull;
    return;
  }
  __shared__ int wsum[L_START_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int base = 0;
  for (int t0 = 0; t0 < L.nseg; t0 += 4 * L_START_THREADS) {
    const int s0 = t0 + 4 * (int)threadIdx.x;
    unsigned on = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (s0 + k < L.nseg && L.cnt[s0 + k] > 0) on |= 1u << k;
    const int n = __popc(on);
    int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    const int w = wsum[lane];  // 32 warps, a sum a lane
    const int before = __reduce_add_sync(0xffffffffu, lane < warp ? w : 0);
    const int all = __reduce_add_sync(0xffffffffu, w);
    int at = base + before + incl - n;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if ((on >> k) & 1u) active[at++] = s0 + k;
    base += all;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    ci[LC_ACTIVE] = base;
    ci[LC_ACC] = ci[LC_SWAP_ITEMS] = ci[LC_COL_ITEMS] = 0;
  }
}

__global__ void k_l_iota2(int* orig, int* pos, int R) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < R; i += gridDim.x * blockDim.x) orig[i] = pos[i] = i;
}

// ---------------------------------------------------------------------------
// Candidates and features
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned mix32(unsigned x) {
  x ^= x >> 16;
  x *= 0x7feb352du;
  x ^= x >> 15;
  x *= 0x846ca68bu;
  x ^= x >> 16;
  return x;
}

// target segment q of segment p in round `round` (never p itself)
__device__ __forceinline__ int target_of(int p, int q, int round, int nseg, unsigned seed) {
  const unsigned h = mix32((unsigned)p * 0x9e3779b9u ^ mix32((unsigned)q + 0x632be5abu * (unsigned)round) ^ seed);
  int t = (int)(h % (unsigned)(nseg - 1));
  return t >= p ? t + 1 : t;
}

// candidate c of segment p: target slot q, offsets i (in p) and j (in t)
__device__ __forceinline__ void cand_of(int c, int M, int& q, int& i, int& j) {
  q = c / (M * M);
  i = (c / M) % M;
  j = c % M;
}

__device__ void features(const LMat& L, int p, int i, int t, int j, float* f) {
  const int u = L.orig[p * L.M + i], w = L.orig[t * L.M + j];
  const int du = L.cptr[u + 1] - L.cptr[u], dw = L.cptr[w + 1] - L.cptr[w];
  const float iu = 1.0f / (float)max(du, 1), iw = 1.0f / (float)max(dw, 1), iR = 1.0f / (float)L.R;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    f[k] = (k + 1 <= L.M) ? L.colh[u * 9 + k + 1] * iu : 0.f;
    f[8 + k] = (k + 1 <= L.M) ? L.colh[w * 9 + k + 1] * iw : 0.f;
  }
#pragma unroll
  for (int k = 0; k < 9; ++k) f[16 + k] = L.hist[t * 9 + k] * iR;
  f[25] = log2f(1.0f + du) * (1.0f / 16);
  f[26] = log2f(1.0f + dw) * (1.0f / 16);
  f[27] = L.hist[p * 9 + L.N] * iR;
  f[28] = L.hist[p * 9 + L.N + 1] * iR;
  f[29] = L.colh[u * 9 + L.N + 1] * (1.0f / 16);
  f[30] = L.colh[w * 9 + L.N + 1] * (1.0f / 16);
  f[31] = 1.0f;
}

// Exact gain of exchanging the columns at positions p*M+i and t*M+j, from
// the group table.  A row holding exactly one of the two columns moves one
// bit between its groups in p and t; a row holding both (or neither) keeps
// its groups.  Objective 0 counts invalid groups (popcount > N) removed,
// objective 1 the nonzeros an N:M pruning keeps (sum of min(popcount, N)).
__device__ __forceinline__ int move_gain(int obj, int N, int from, int to) {  // popcounts before the move
  return obj == 0 ? (from == N + 1) - (to == N) : (to < N) - (from <= N);
}

// The rows of both columns are one list, 8 a lane in flight, and the next
// ones' numbers are fetched while the group bytes come: a hub column's rows
// are a long chain of dependent loads on one warp.  (4 a lane, column after
// column and without the fetch ahead, eleven rounds at 65536 rows: 618 us,
// 447 now.)
__device__ int exact_gain_warp(const LMat& L, int p, int i, int t, int j) {
  constexpr int U = 8;
  const int lane = threadIdx.x & 31;
  const int u = L.orig[p * L.M + i], w = L.orig[t * L.M + j];
  const unsigned bi = 1u << i, bj = 1u << j;
  const int bu = L.cptr[u], du = L.cptr[u + 1] - bu, bw = L.cptr[w], n = du + L.cptr[w + 1] - bw;
  auto row = [&](int e) { return e < du ? L.crow[bu + e] : e < n ? L.crow[bw + e - du] : -1; };
  int r[U];
#pragma unroll
  for (int k = 0; k < U; ++k) r[k] = row(lane + 32 * k);
  int g = 0;
  for (int e0 = lane; e0 - lane < n; e0 += 32 * U) {
    unsigned gp[U], gt[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      gp[k] = r[k] >= 0 ? L.G[(long long)r[k] * L.nseg + p] : 0u;
      gt[k] = r[k] >= 0 ? L.G[(long long)r[k] * L.nseg + t] : 0u;
    }
    int next[U];
#pragma unroll
    for (int k = 0; k < U; ++k) next[k] = row(e0 + 32 * (U + k));
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const bool first = e0 + 32 * k < du;  // a row of column u, else of column w
      const unsigned from = first ? gp[k] : gt[k], to = first ? gt[k] : gp[k];
      if (r[k] >= 0 && !(to & (first ? bj : bi)))  // else both columns are here
        g += move_gain(L.obj, L.N, __popc(from), __popc(to));
      r[k] = next[k];
    }
  }
  return __reduce_add_sync(0xffffffffu, g);
}

// ---------------------------------------------------------------------------
// MLP inference on tcgen05 (fused with feature construction and top-8)
// ---------------------------------------------------------------------------
struct MlpW {  // device weights
  const float* W1;  // [LH][LF]
  const float* b1;  // [LH]
  const float* W2;  // [LH][LH]
  const float* b2;
  const float* w3;  // [LH]
  const float* b3;  // [1]
};

// K-major canonical layout of a [rows x K] bf16 operand: core matrices of
// 8 rows x 16 bytes; k-chunks at 128 B, 8-row groups at K*16 B.
__device__ __forceinline__ int kmaj_off(int r, int k, int K) {
  return (r >> 3) * (K * 16) + (k >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2;
}

// A block is four groups of 128 threads with a tile of 128 candidates each in
// flight, on one copy of the weights.
constexpr int MG = 4;              // groups a block
constexpr int ML_THREADS = MG * 128;
// Staged columns of a tile: its target slots' (at most 32 slots, 64 columns),
// the segment's own from ML_OWN on.
constexpr int ML_OWN = 72, ML_COLS = ML_OWN + 8, ML_SLOTS = 32;

struct MlpGroup {
  alignas(1024) unsigned char A[128 * LH * 2];  // a tile's features (8 KB of it), then its first layer's output
  unsigned key[2048];                            // the segment's scores, order-preserving (0: NaN)
  uint4 colf[ML_COLS], slotf[ML_SLOTS];          // features of a column or a slot in BF16: eight of the histogram
  unsigned colx[ML_COLS], slotx[ML_SLOTS];       // ... and the rest: degree | N+1 rows << 16; ninth of the histogram
  unsigned own;                                  // the segment's two features
};
struct MlpSmem {
  alignas(1024) unsigned char W1[LH * LF * 2];  // 8 KB
  alignas(1024) unsigned char W2[LH * LH * 2];  // 32 KB
  MlpGroup g[MG];                               // 42 KB each
  float b1[LH], b2[LH], w3[LH];                 // plain mode
  alignas(8) uint64_t bar[MG];
  uint32_t tmem;
  int err;
};

// The biases and the last layer as a kernel argument: read in unrolled code
// they are operands from the constant bank.
struct MlpTail {
  float b1[LH];
  float b2[LH], w3[LH], b3;  // as in the parameter vector
};

__device__ __forceinline__ void fence_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void group_sync(int g) { asm volatile("bar.sync %0, 128;" ::"r"(g + 1) : "memory"); }
__device__ __forceinline__ unsigned bf2(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const unsigned*>(&h);
}
// ReLU of two values, rounded to BF16: as rounding the ReLU, for NaN (0) too
__device__ __forceinline__ unsigned relu_bf2(float lo, float hi) {
  const __nv_bfloat162 h = __hmax2(__floats2bfloat162_rn(lo, hi), __floats2bfloat162_rn(0.f, 0.f));
  return *reinterpret_cast<const unsigned*>(&h);
}

// The MLP on tcgen05.  Candidate mode (kPlain = false): a group takes an active
// segment at a time, scores all of its candidates and keeps the best LTOP ids
// in top[a], at most one per target segment (ties to the lower id), so the
// exactly scored proposals are not near-copies of one swap.  Plain mode: rows
// of X in tiles of 128, scores to Y (the inference path on given features, for
// tests and timing).  Per tile: features -> A (bf16, K-major), MMA 128x128x32
// into the group's 128 tensor-memory columns, bias + ReLU -> A, MMA
// 128x128x128 into the same columns, bias + ReLU + dot with w3 in registers in
// ascending order.  Thread t owns candidate t of the tile, which is TMEM lane
// t.
//
// Bound by issue: some 800 instructions a warp and tile, four warps to a
// scheduler.  What made the form before this one (a group a block, two blocks
// an SM) 2.5 times slower was the shared-memory pipe: the biases and w3 read
// by every thread (an LDS costs a cycle for 32 lanes' word, broadcast or not),
// first-layer stores of 4 bytes with four-way conflicts, and every candidate
// making all of its features.  Now the biases come from the constant bank, a
// thread stores 16 bytes of its row at a time (eight lanes' pieces are
// contiguous), and a column's or slot's features are made once a tile by one
// thread and copied.  At 8192 segments x 256 candidates: 176 -> 58 us.
template <bool kPlain>
__global__ void __launch_bounds__(ML_THREADS, 1)
    k_l_mlp(LMat L, MlpW W, const __grid_constant__ MlpTail T, const int* active, const int* nactive_p, int KT,
            int round, unsigned seed, int* top, const float* X, int nX, float* Y, int* err) {
  extern __shared__ unsigned char l_raw[];
  MlpSmem& sm = *reinterpret_cast<MlpSmem*>(
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(l_raw) + 1023) & ~uintptr_t(1023)));
  const int tid = threadIdx.x, g = tid >> 7, t = tid & 127;
  const int warp = tid >> 5, lane = tid & 31;
  const int nwork = kPlain ? (nX + 127) / 128 : *nactive_p;
  if ((int)blockIdx.x >= nwork) return;
  // weights -> canonical layouts (B operands: rows = output features, K-major), 16 bytes at a time
  auto weights = [&](const float* w, unsigned char* dst, int K) {
    for (int e = tid; e < LH * K / 8; e += ML_THREADS) {
      float x[8];  // (the parameter vector is 4-byte aligned only where a layer starts)
#pragma unroll
      for (int z = 0; z < 8; ++z) x[z] = w[8 * e + z];
      const int n = 8 * e / K, k = 8 * e % K;
      *reinterpret_cast<uint4*>(dst + kmaj_off(n, k, K)) =
          make_uint4(bf2(x[0], x[1]), bf2(x[2], x[3]), bf2(x[4], x[5]), bf2(x[6], x[7]));
    }
  };
  weights(W.W1, sm.W1, LF);
  weights(W.W2, sm.W2, LH);
  if (kPlain)
    for (int e = tid; e < LH; e += ML_THREADS) {
      sm.b1[e] = W.b1[e];
      sm.b2[e] = W.b2[e];
      sm.w3[e] = W.w3[e];
    }
  if (tid == 0) {
    for (int k = 0; k < MG; ++k) ptx::mbar_init(&sm.bar[k], 1);
    sm.err = 0;
    ptx::fence_mbar_init();
  }
  if (warp == 0) {
    ptx::tmem_alloc(&sm.tmem, MG * LH);
    ptx::tmem_relinquish();
  }
  fence_async_smem();
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  MlpGroup& G = sm.g[g];
  uint64_t* const bar = &sm.bar[g];
  const uint32_t tm = sm.tmem + (uint32_t)(g * LH), tl = tm + ((uint32_t)((warp & 3) * 32) << 16);
  const uint32_t idesc = ptx::idesc_f16(1u, 0u, 0u, 128, LH);
  const float b3 = kPlain ? W.b3[0] : T.b3;
  const int MM = L.M * L.M;
  const int ncand = kPlain ? 0 : KT * MM;
  const int ntile = kPlain ? 1 : (ncand + 127) / 128;
  const int step = MG * gridDim.x;
  uint32_t phase = 0;
  // What this thread makes of tile (a, tile)'s features: of one column (v, x),
  // one slot (v, x), the segment's two (x), or in plain mode its row's.  The
  // next tile's are loaded while the tensor core runs the current one's first
  // layer, so their loads' latency is hidden behind it.
  uint4 v = make_uint4(0u, 0u, 0u, 0u);
  unsigned x = 0u;
  float f[kPlain ? LF : 1];
  auto load = [&](int a, int tile) {
    if (a >= nwork) return;
    if constexpr (kPlain) {
      const int c = a * 128 + t;
#pragma unroll
      for (int k = 0; k < LF; ++k) f[k] = c < nX ? X[(size_t)c * LF + k] : 0.f;
    } else {
      const int p = active[a], slot0 = tile * 128 / MM;
      const int nslot = (min(ncand, tile * 128 + 128) - 1) / MM - slot0 + 1;
      const float iR = 1.0f / (float)L.R;
      int at = -1;  // position of this thread's column
      if (t < nslot * L.M) at = target_of(p, slot0 + t / L.M, round, L.nseg, seed) * L.M + t % L.M;
      else if (t >= ML_OWN && t < ML_OWN + L.M && tile == 0) at = p * L.M + t - ML_OWN;
      if (at >= 0) {
        const int u = L.orig[at], d = L.cptr[u + 1] - L.cptr[u];
        const float id = 1.0f / (float)max(d, 1);
        float h[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) h[k] = k + 1 <= L.M ? L.colh[u * 9 + k + 1] * id : 0.f;
        v = make_uint4(bf2(h[0], h[1]), bf2(h[2], h[3]), bf2(h[4], h[5]), bf2(h[6], h[7]));
        x = bf2(log2f(1.0f + d) * (1.0f / 16), L.colh[u * 9 + L.N + 1] * (1.0f / 16));
      } else if (t >= ML_COLS && t < ML_COLS + nslot) {
        const int* hs = L.hist + (size_t)target_of(p, slot0 + t - ML_COLS, round, L.nseg, seed) * 9;
        float h[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) h[k] = hs[k] * iR;
        v = make_uint4(bf2(h[0], h[1]), bf2(h[2], h[3]), bf2(h[4], h[5]), bf2(h[6], h[7]));
        x = bf2(h[8], 0.f);
      } else if (t == 127) {
        x = bf2(L.hist[p * 9 + L.N] * iR, L.hist[p * 9 + L.N + 1] * iR);
      }
    }
  };
  const int a0 = g * gridDim.x + blockIdx.x;
  load(a0, 0);
  for (int a = a0; a < nwork; a += step) {
    for (int tile = 0; tile < ntile; ++tile) {
      const int c = kPlain ? a * 128 + t : tile * 128 + t;
      const bool live = kPlain ? c < nX : c < ncand;
      // (A: the second layer of the tile before has read it, as every thread
      // has waited for; the staged features: read before the barrier that
      // followed)
      uint4 row[4];
      if constexpr (kPlain) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          row[k] = make_uint4(bf2(f[8 * k], f[8 * k + 1]), bf2(f[8 * k + 2], f[8 * k + 3]),
                              bf2(f[8 * k + 4], f[8 * k + 5]), bf2(f[8 * k + 6], f[8 * k + 7]));
      } else {
        const int slot0 = tile * 128 / MM;
        const int nslot = (min(ncand, tile * 128 + 128) - 1) / MM - slot0 + 1;
        if (t < nslot * L.M || (t >= ML_OWN && t < ML_OWN + L.M && tile == 0)) {
          G.colf[t] = v;
          G.colx[t] = x;
        } else if (t >= ML_COLS && t < ML_COLS + nslot) {
          G.slotf[t - ML_COLS] = v;
          G.slotx[t - ML_COLS] = x;
        } else if (t == 127) {
          G.own = x;
        }
        group_sync(g);
#pragma unroll
        for (int k = 0; k < 4; ++k) row[k] = make_uint4(0u, 0u, 0u, 0u);
        if (live) {
          int q, i, j;
          cand_of(c, L.M, q, i, j);
          const int z = q - slot0, w = z * L.M + j;
          const unsigned xu = G.colx[ML_OWN + i], xw = G.colx[w], xp = G.own;
          row[0] = G.colf[ML_OWN + i];
          row[1] = G.colf[w];
          row[2] = G.slotf[z];
          row[3] = make_uint4((G.slotx[z] & 0xffffu) | xu << 16, (xw & 0xffffu) | xp << 16,
                              xp >> 16 | (xu & 0xffff0000u), xw >> 16 | bf2(0.f, 1.f));
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) *reinterpret_cast<uint4*>(G.A + kmaj_off(t, 8 * k, LF)) = row[k];
      fence_async_smem();
      ptx::tc_fence_before();
      group_sync(g);
      ptx::tc_fence_after();
      if (t == 0) {
        for (int kk = 0; kk < LF / 16; ++kk) {
          const uint64_t ad = ptx::smem_desc(ptx::smem_addr(G.A) + kk * 256, 128, LF * 16, 0);
          const uint64_t bd = ptx::smem_desc(ptx::smem_addr(sm.W1) + kk * 256, 128, LF * 16, 0);
          ptx::mma_f16(tm, ad, bd, idesc, kk > 0 ? 1u : 0u);
        }
        ptx::mma_commit(bar);
      }
      if (tile + 1 < ntile) load(a, tile + 1);
      else load(a + step, 0);
      if (!ptx::mbar_wait(bar, phase, L_WAIT)) sm.err = 1;
      phase ^= 1u;
      ptx::tc_fence_after();
      // layer 1 epilogue: bias, ReLU, BF16 -> A (the first layer has read it)
#pragma unroll
      for (int c0 = 0; c0 < LH; c0 += 32) {
        uint32_t d[32];
        ptx::tmem_ld_32x32b_x32(tl + (uint32_t)c0, d);
        ptx::tmem_ld_wait();
        auto b = [&](int z) { return kPlain ? sm.b1[c0 + z] : T.b1[c0 + z]; };
        auto h = [&](int z) {
          return relu_bf2(__uint_as_float(d[z]) + b(z), __uint_as_float(d[z + 1]) + b(z + 1));
        };
#pragma unroll
        for (int z = 0; z < 32; z += 8)
          *reinterpret_cast<uint4*>(G.A + kmaj_off(t, c0 + z, LH)) = make_uint4(h(z), h(z + 2), h(z + 4), h(z + 6));
      }
      fence_async_smem();
      ptx::tc_fence_before();
      group_sync(g);
      ptx::tc_fence_after();
      if (t == 0) {
        for (int kk = 0; kk < LH / 16; ++kk) {
          const uint64_t ad = ptx::smem_desc(ptx::smem_addr(G.A) + kk * 256, 128, LH * 16, 0);
          const uint64_t bd = ptx::smem_desc(ptx::smem_addr(sm.W2) + kk * 256, 128, LH * 16, 0);
          ptx::mma_f16(tm, ad, bd, idesc, kk > 0 ? 1u : 0u);
        }
        ptx::mma_commit(bar);
      }
      if (!ptx::mbar_wait(bar, phase, L_WAIT)) sm.err = 1;
      phase ^= 1u;
      ptx::tc_fence_after();
      float y = b3;
#pragma unroll
      for (int c0 = 0; c0 < LH; c0 += 32) {
        uint32_t d[32];
        ptx::tmem_ld_32x32b_x32(tl + (uint32_t)c0, d);
        ptx::tmem_ld_wait();
        auto b = [&](int z) { return kPlain ? sm.b2[c0 + z] : T.b2[c0 + z]; };
        auto w3 = [&](int z) { return kPlain ? sm.w3[c0 + z] : T.w3[c0 + z]; };
#pragma unroll
        for (int z = 0; z < 32; z += 2) {
          const unsigned h = relu_bf2(__uint_as_float(d[z]) + b(z), __uint_as_float(d[z + 1]) + b(z + 1));
          y = fmaf(__uint_as_float(h << 16), w3(z), y);
          y = fmaf(__uint_as_float(h & 0xffff0000u), w3(z + 1), y);
        }
      }
      if (kPlain) {
        if (live) Y[c] = y;
      } else if (live) {
        const unsigned bits = __float_as_uint(y + 0.f);  // (-0 equals 0)
        G.key[c] = y != y ? 0u : (bits >> 31 ? ~bits : bits | 0x80000000u);
      }
    }
    if (!kPlain) {
      // top LTOP of this segment (ties to the lower id); the group's first
      // warp (the others write scores again only past barriers that it joins)
      group_sync(g);
      if (t < 32) {
        const unsigned dropped = ~0xff800000u;  // the key of -infinity
        for (int k = 0; k < LTOP; ++k) {
          unsigned best = 0u;
          int bid = 0x7fffffff;
          for (int c = lane; c < ncand; c += 32) {
            const unsigned s = G.key[c];
            if (s > best) {
              best = s;
              bid = c;
            }
          }
          const unsigned m = __reduce_max_sync(0xffffffffu, best);
          bid = __reduce_min_sync(0xffffffffu, m != 0u && best == m ? bid : 0x7fffffff);
          if (lane == 0) top[a * LTOP + k] = bid < ncand ? bid : -1;
          // one proposal per target segment: drop the rest of the winner's slot
          if (bid < ncand) {
            const int q0 = bid / MM;
            for (int z = lane; z < MM; z += 32) G.key[q0 * MM + z] = dropped;
          }
          __syncwarp();
        }
      }
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  if (tid == 0 && sm.err) atomicOr(err, 8);
  if (warp == 0) ptx::tmem_dealloc(sm.tmem, MG * LH);
}

// ---------------------------------------------------------------------------
// Exact scoring, matching, apply
// ---------------------------------------------------------------------------
enum { L_MODE_MLP = 0, L_MODE_EXHAUSTIVE = 1, L_MODE_RANDOM = 2 };

// Exact gains of candidates: the first topk (<= LTOP) proposals of each
// active segment (network or random), or every candidate (exhaustive).  Each active
// segment's best strictly positive candidate goes to best[a] as
// (gain << 40 | (2^40 - 1 - candidate)), so larger is better and ties go to
// the lower candidate id; 0 when none improves.  A sample of the scored
// candidates (1 in dump_every) is written out as (features, gain) pairs.
__global__ void k_l_exact(LMat L, const int* active, const int* nactive_p, int KT, int round, unsigned seed,
                          const int* top, int mode, int topk, unsigned long long* best, float* dump_x, float* dump_y,
                          int dump_every, int* ndump, int dump_cap, unsigned long long* nscored) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  const int nactive = *nactive_p;
  const int ncand = KT * L.M * L.M;
  const int per = mode == L_MODE_EXHAUSTIVE ? ncand : topk;
  unsigned long long scored = 0;
  for (long long w = warp; w < (long long)nactive * per; w += nw) {
    const int a = (int)(w / per), k = (int)(w % per);
    int c;
    if (mode == L_MODE_EXHAUSTIVE) c = k;
    else if (mode == L_MODE_RANDOM) c = (int)(mix32((unsigned)w * 0x9e3779b9u ^ mix32((unsigned)round ^ seed)) % (unsigned)ncand);
    else c = top[a * LTOP + k];
    if (c < 0) continue;
    const int p = active[a];
    int q, i, j;
    cand_of(c, L.M, q, i, j);
    const int t = target_of(p, q, round, L.nseg, seed);
    const int g = exact_gain_warp(L, p, i, t, j);
    ++scored;
    if (lane == 0) {
      if (g > 0)
        atomicMax(&best[a], ((unsigned long long)g << 40) | ((1ull << 40) - 1 - (unsigned long long)c));
      if (dump_x && dump_every > 0 &&
          (mix32((unsigned)w * 2654435761u ^ seed ^ mix32((unsigned)round)) % (unsigned)dump_every) == 0) {
        const int slot = atomicAdd(ndump, 1);
        if (slot < dump_cap) {
          float f[LF];
          features(L, p, i, t, j, f);
          for (int z = 0; z < LF; ++z) dump_x[(size_t)slot * LF + z] = f[z];
          dump_y[slot] = (float)g;
        }
      }
    }
  }
  if (lane == 0 && scored) atomicAdd(nscored, scored);
}

// claim both segments of each segment's best swap; the highest claim wins
__global__ void k_l_claim(LMat L, const int* active, const int* nactive_p, int round, unsigned seed,
                          const unsigned long long* best, unsigned long long* claim) {
  const int nactive = *nactive_p;
  for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < nactive; a += gridDim.x * blockDim.x) {
    const unsigned long long b = best[a];
    if (!b) continue;
    const int c = (int)((1ull << 40) - 1 - (b & ((1ull << 40) - 1)));
    int q, i, j;
    cand_of(c, L.M, q, i, j);
    const int p = active[a], t = target_of(p, q, round, L.nseg, seed);
    const unsigned long long key = (b & ~((1ull << 40) - 1)) | (unsigned long long)(unsigned)a;
    atomicMax(&claim[p], key);
    atomicMax(&claim[t], key);
  }
}

// Winners: swaps that hold the claim on both of their segments, so accepted
// swaps touch disjoint segments and their exact gains add up.  A winner's
// nodes exchange places here, and the chunks of its two columns go to the
// work list of k_l_apply_rows as (swap, chunk), the first column's first.
__global__ void k_l_accept(LMat L, const int* active, int* ci, int round, unsigned seed,
                           const unsigned long long* best, const unsigned long long* claim, int4* acc, int2* uw,
                           int2* items, unsigned long long* gain_sum) {
  const int nactive = ci[LC_ACTIVE], lane = threadIdx.x & 31;
  for (int a0 = blockIdx.x * blockDim.x + threadIdx.x - lane; a0 < nactive; a0 += gridDim.x * blockDim.x) {
    const int a = a0 + lane;
    const unsigned long long b = a < nactive ? best[a] : 0ull;
    int n = 0, nitems = 0;
    int4 sw;
    int2 nodes;
    if (b) {
      const int c = (int)((1ull << 40) - 1 - (b & ((1ull << 40) - 1)));
      int q, i, j;
      cand_of(c, L.M, q, i, j);
      const int p = active[a], t = target_of(p, q, round, L.nseg, seed);
      const unsigned long long key = (b & ~((1ull << 40) - 1)) | (unsigned long long)(unsigned)a;
      if (claim[p] == key && claim[t] == key) {
        n = 1;
        sw = make_int4(p, i, t, j);
        const int x = p * L.M + i, y = t * L.M + j;
        const int u = L.orig[x], w = L.orig[y];
        nodes = make_int2(u, w);
        nitems = chunks_of(L, u) + chunks_of(L, w);
        L.orig[x] = w;
        L.orig[y] = u;
        L.pos[w] = x;
        L.pos[u] = y;
        atomicAdd(gain_sum, b >> 40);
      }
    }
    const int s = warp_append(n, ci + LC_ACC), at = warp_append(nitems, ci + LC_SWAP_ITEMS);
    if (n) {
      acc[s] = sw;
      uw[s] = nodes;
      for (int k = 0; k < nitems; ++k) items[at + k] = make_int2(s, k);
    }
  }
}

// Apply accepted swaps: flip the two bits of every row that holds exactly one
// of the two columns and keep hist / cnt in step.  Accepted swaps touch
// disjoint segments, and a row holding both columns moves nothing, so the
// rows of the two columns are independent: they are cut into chunks of
// L_CHUNK, one warp a chunk, which sums its hist / cnt changes in registers
// and adds them once.  The columns of the swaps' segments are listed for
// their new histograms on the side: that reads nothing that changes here.
__global__ void k_l_apply_rows(LMat L, const int4* acc, int* ci, const int2* uw, const int2* items,
                               int2* col_items) {
  const int n = ci[LC_ACC], tot = ci[LC_SWAP_ITEMS];
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  for (int e0 = 32 * warp; e0 < n * 2 * L.M; e0 += 32 * nw) {  // n * 2M <= R
    const int e = e0 + lane;
    const bool live = e < n * 2 * L.M;
    int a = 0;
    if (live) {
      const int4 sw = acc[e / (2 * L.M)];
      const int k = e % (2 * L.M);
      a = (k < L.M ? sw.x : sw.z) * L.M + k % L.M;
    }
    take_column(L, a, live, col_items, ci + LC_COL_ITEMS);
  }
  unsigned* Gw = reinterpret_cast<unsigned*>(L.G);
  for (int item = warp; item < tot; item += nw) {
    const int s = items[item].x;
    const int4 sw = acc[s];
    const int p = sw.x, i = sw.y, t = sw.z, j = sw.w;
    const int u = uw[s].x, w = uw[s].y;
    const unsigned bi = 1u << i, bj = 1u << j;
    const int cu = chunks_of(L, u);
    int k = items[item].y;
    const int col = k < cu ? u : w;
    if (k >= cu) k -= cu;
    const int beg = L.cptr[col] + k * L_CHUNK, end = min(beg + L_CHUNK, L.cptr[col + 1]);
    int dp[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, dt[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    int dcp = 0, dct = 0;
    int r[L_ROWS];
    unsigned was_p[L_ROWS], was_t[L_ROWS];
#pragma unroll
    for (int x = 0; x < L_ROWS; ++x) r[x] = beg + lane + 32 * x < end ? L.crow[beg + lane + 32 * x] : -1;
#pragma unroll
    for (int x = 0; x < L_ROWS; ++x) {
      was_p[x] = r[x] >= 0 ? L.G[(long long)r[x] * L.nseg + p] : 0u;
      was_t[x] = r[x] >= 0 ? L.G[(long long)r[x] * L.nseg + t] : 0u;
    }
#pragma unroll
    for (int x = 0; x < L_ROWS; ++x) {
      const long long cp = (long long)r[x] * L.nseg + p, ct = (long long)r[x] * L.nseg + t;
      const unsigned gp = was_p[x], gt = was_t[x];  // (no row: both 0, nothing moves)
      const bool inU = gp & bi, inW = gt & bj;
      if (inU == inW) continue;  // both columns or neither: nothing moves
      const unsigned np_ = inW ? (gp | bi) : (gp & ~bi);
      const unsigned nt_ = inU ? (gt | bj) : (gt & ~bj);
      atomicXor(&Gw[cp >> 2], (gp ^ np_) << ((cp & 3) * 8));
      atomicXor(&Gw[ct >> 2], (gt ^ nt_) << ((ct & 3) * 8));
      const int a0 = __popc(gp), a1 = __popc(np_), c0 = __popc(gt), c1 = __popc(nt_);
#pragma unroll
      for (int z = 0; z < 9; ++z) {
        dp[z] += (z == a1) - (z == a0);
        dt[z] += (z == c1) - (z == c0);
      }
      dcp += (a1 > L.N) - (a0 > L.N);
      dct += (c1 > L.N) - (c0 > L.N);
    }
#pragma unroll
    for (int z = 0; z < 9; ++z) {
      const int vp = __reduce_add_sync(0xffffffffu, dp[z]), vt = __reduce_add_sync(0xffffffffu, dt[z]);
      if (lane == z && vp) atomicAdd(&L.hist[p * 9 + z], vp);
      if (lane == z && vt) atomicAdd(&L.hist[t * 9 + z], vt);
    }
    const int vcp = __reduce_add_sync(0xffffffffu, dcp), vct = __reduce_add_sync(0xffffffffu, dct);
    if (lane == 0 && vcp) atomicAdd(&L.cnt[p], vcp);
    if (lane == 0 && vct) atomicAdd(&L.cnt[t], vct);
  }
}

// totals from the segment histograms: [0] invalid groups, [1] retained nonzeros
__global__ void k_l_totals(const int* hist, int nseg, int N, unsigned long long* out) {
  unsigned long long inv = 0, ret = 0;
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < nseg; s += gridDim.x * blockDim.x)
    for (int k = 1; k <= 8; ++k) {
      const unsigned long long h = (unsigned long long)hist[s * 9 + k];
      if (k > N) inv += h;
      ret += h * (unsigned long long)(k < N ? k : N);
    }
  for (int o = 16; o > 0; o >>= 1) {
    inv += __shfl_xor_sync(0xffffffffu, inv, o);
    ret += __shfl_xor_sync(0xffffffffu, ret, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&out[0], inv);
    atomicAdd(&out[1], ret);
  }
}

__global__ void k_l_invert(const int* orig, int R, int* newpos) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < R; i += gridDim.x * blockDim.x) newpos[orig[i]] = i;
}

}  // namespace vnm

// ---------------------------------------------------------------------------
// Training kernels (FP32 accumulation; operands rounded to BF16 exactly where
// the tensor-core inference rounds them: the layer inputs and the weights).
// An Adam step is two kernels:
//   k_t_rows   everything that belongs to one batch row: both layers, the
//              output and its error, and the errors of the hidden layers;
//   k_t_wgrad  the sums over the batch, and Adam on the sums it made.
// Every sum runs over its index in ascending order in one FP32 chain, so the
// results do not depend on the tiling.  At 1024 rows a step takes 18 us (one
// thread per output over global memory, nine launches: 0.5 ms).
// ---------------------------------------------------------------------------
namespace vnm {

__device__ __forceinline__ float bf(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// The hidden layers' weights rounded to BF16, rows padded by 16 bytes: a warp
// reads 8 rows' 16-byte pieces, or 32 consecutive words, without bank
// conflicts.  Kept in global memory in the form that k_t_rows copies to
// shared memory (made by k_t_round, kept up by Adam).
struct TrainW {
  float W1[LH][LF + 4];
  float W2[LH][LH + 4];
};

// What a step's rows leave for the sums over the batch, transposed so that a
// unit's values of consecutive rows are contiguous; ld = the batch rounded up
// to 16 rows, the rows past the batch zero.
struct TrainActs {
  float* X;    // [LF][ld] inputs, rounded to BF16 like the layers
  float* H1;   // [LH][ld] first hidden layer
  float* H2;   // [LH][ld] second
  float* dZ1;  // [LH][ld] dL / d(first layer before the ReLU)
  float* dZ2;  // [LH][ld]
  float* dy;   // [ld]
  TrainW* W;
  int ld;
};

__global__ void k_t_round(const float* W1, const float* W2, TrainW* W) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < LH * (LF + 4 + LH + 4); e += gridDim.x * blockDim.x) {
    if (e < LH * (LF + 4)) {
      const int o = e / (LF + 4), i = e % (LF + 4);
      W->W1[o][i] = i < LF ? bf(W1[o * LF + i]) : 0.f;
    } else {
      const int o = (e - LH * (LF + 4)) / (LH + 4), i = (e - LH * (LF + 4)) % (LH + 4);
      W->W2[o][i] = i < LH ? bf(W2[o * LH + i]) : 0.f;
    }
  }
}

// 8 rows a block (a 1024-row batch on 128 of the 152 SMs); a thread has 2
// units of both hidden layers for 4 of the rows.  Bound by the words read
// from shared memory, a 4-byte word a lane costing the SM a cycle whether or
// not lanes share it: 6 words for 8 FMAs on each of 4 warps.  The 128-deep layer forward
// takes 3.5 K cycles; one unit a thread on 8 warps (5 words for 4 FMAs) took
// 7.5 K, 4 units on 2 warps, bound by their issue rate, 4.4 K.
constexpr int T_ROWS = 8, T_U = 2, T_US = LH / T_U;  // a thread's units are T_US apart
constexpr int T_THREADS = T_US * (T_ROWS / 4);
struct TrainRowsSmem {
  TrainW W;
  alignas(16) float x[LF][T_ROWS];
  alignas(16) float h1[LH][T_ROWS];
  alignas(16) float h2[LH][T_ROWS];
  alignas(16) float d2[LH][T_ROWS];
  alignas(16) float w3[LH];
  float dy[T_ROWS];
};

// s[j][r] = sum_k a[k][r] * w_j[k] for T_U units j and 4 rows r, k ascending in
// one chain each, two rows to a packed FMA (two round-to-nearest FMAs).
// kByRow: unit j's weights are a row of W (w[j * T_US * pitch + k]), else a
// column (w[k * pitch + j * T_US]).  Four k's operands are loaded while the
// four before them are summed.
template <int N, int PITCH, bool kByRow>
__device__ __forceinline__ void dot_rows(const float* a, const float* w, float (&s)[T_U][4]) {
  unsigned long long s01[T_U], s23[T_U];
#pragma unroll
  for (int j = 0; j < T_U; ++j) s01[j] = s23[j] = 0ull;
  float wk[2][T_U][4];
  ulonglong2 v[2][4];
  auto fetch = [&](int k0, int h) {
#pragma unroll
    for (int j = 0; j < T_U; ++j) {
      if (kByRow) {
        const float4 q = *reinterpret_cast<const float4*>(w + j * T_US * PITCH + k0);
        wk[h][j][0] = q.x;
        wk[h][j][1] = q.y;
        wk[h][j][2] = q.z;
        wk[h][j][3] = q.w;
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) wk[h][j][k] = w[(k0 + k) * PITCH + j * T_US];
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) v[h][k] = *reinterpret_cast<const ulonglong2*>(a + (k0 + k) * T_ROWS);
  };
  auto add = [&](int h) {
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int j = 0; j < T_U; ++j) {
        unsigned long long ww;
        asm("mov.b64 %0, {%1, %1};" : "=l"(ww) : "r"(__float_as_uint(wk[h][j][k])));
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(s01[j]) : "l"(v[h][k].x), "l"(ww));
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(s23[j]) : "l"(v[h][k].y), "l"(ww));
      }
  };
  fetch(0, 0);
#pragma unroll 1
  for (int k0 = 0; k0 < N; k0 += 8) {
    fetch(k0 + 4, 1);
    add(0);
    if (k0 + 8 < N) fetch(k0 + 8, 0);
    add(1);
  }
#pragma unroll
  for (int j = 0; j < T_U; ++j) {
    s[j][0] = __uint_as_float((uint32_t)s01[j]);
    s[j][1] = __uint_as_float((uint32_t)(s01[j] >> 32));
    s[j][2] = __uint_as_float((uint32_t)s23[j]);
    s[j][3] = __uint_as_float((uint32_t)(s23[j] >> 32));
  }
}

__global__ void __launch_bounds__(T_THREADS) k_t_rows(const float* __restrict__ X, const float* __restrict__ t, int B,
                                                      MlpW W, TrainActs A, float* loss) {
  extern __shared__ __align__(16) unsigned char t_raw[];
  TrainRowsSmem& sm = *reinterpret_cast<TrainRowsSmem*>(t_raw);
  const int tid = threadIdx.x, u0 = tid % T_US, r0 = (tid / T_US) * 4;  // this thread's first unit and first row
  const int b0 = blockIdx.x * T_ROWS, live = min(T_ROWS, B - b0);
  ptx::grid_dependents_launch();
  ptx::grid_dependency_wait();  // the weights and the activations are the step before's
  for (int e = tid; e < (int)sizeof(TrainW) / 16; e += T_THREADS)
    ptx::cp_async16_zfill(t_raw + e * 16, reinterpret_cast<const unsigned char*>(A.W) + e * 16, 16u);
  ptx::cp_async_commit();
  float b1[T_U], b2[T_U], w3[T_U];
#pragma unroll
  for (int j = 0; j < T_U; ++j) {
    b1[j] = W.b1[u0 + T_US * j];
    b2[j] = W.b2[u0 + T_US * j];
    w3[j] = W.w3[u0 + T_US * j];
    if (r0 == 0) sm.w3[u0 + T_US * j] = w3[j];
  }
  const float b3 = W.b3[0];
  const float target = tid < live ? t[b0 + tid] : 0.f;
  for (int e = tid; e < LF * T_ROWS; e += T_THREADS) {
    const int r = e / LF, k = e % LF;
    sm.x[k][r] = r < live ? bf(X[(size_t)(b0 + r) * LF + k]) : 0.f;
  }
  ptx::cp_async_wait<0>();
  __syncthreads();
  // one layer's activations: kept in z, rounded in h, out to the batch's arrays
  auto finish = [&](float (&z)[T_U][4], const float (&bias)[T_U], float (*h)[T_ROWS], float* out) {
#pragma unroll
    for (int j = 0; j < T_U; ++j) {
      float v[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        z[j][r] = fmaxf(z[j][r] + bias[j], 0.f);
        v[r] = bf(z[j][r]);
      }
      *reinterpret_cast<float4*>(&h[u0 + T_US * j][r0]) = make_float4(v[0], v[1], v[2], v[3]);
#pragma unroll
      for (int r = 0; r < 4; ++r)
        if (r0 + r >= live) v[r] = 0.f;
      *reinterpret_cast<float4*>(out + (size_t)(u0 + T_US * j) * A.ld + b0 + r0) = make_float4(v[0], v[1], v[2], v[3]);
    }
  };
  float z1[T_U][4], z2[T_U][4], d[T_U][4];
  dot_rows<LF, LF + 4, true>(&sm.x[0][r0], sm.W.W1[u0], z1);
  finish(z1, b1, sm.h1, A.H1);
  __syncthreads();
  dot_rows<LH, LH + 4, true>(&sm.h1[0][r0], sm.W.W2[u0], z2);
  finish(z2, b2, sm.h2, A.H2);
  if (u0 < LF)
    *reinterpret_cast<float4*>(A.X + (size_t)u0 * A.ld + b0 + r0) = *reinterpret_cast<const float4*>(&sm.x[u0][r0]);
  __syncthreads();
  if (tid < T_ROWS) {  // the output, its error and the row's part of mean((y - t)^2) / 2
    float s = b3;
#pragma unroll 4
    for (int o = 0; o < LH; o += 8) {
      const float4 wa = *reinterpret_cast<const float4*>(&sm.w3[o]), wb = *reinterpret_cast<const float4*>(&sm.w3[o + 4]);
      s = fmaf(sm.h2[o][tid], wa.x, s);
      s = fmaf(sm.h2[o + 1][tid], wa.y, s);
      s = fmaf(sm.h2[o + 2][tid], wa.z, s);
      s = fmaf(sm.h2[o + 3][tid], wa.w, s);
      s = fmaf(sm.h2[o + 4][tid], wb.x, s);
      s = fmaf(sm.h2[o + 5][tid], wb.y, s);
      s = fmaf(sm.h2[o + 6][tid], wb.z, s);
      s = fmaf(sm.h2[o + 7][tid], wb.w, s);
    }
    float dy = 0.f, l = 0.f;
    if (tid < live) {
      const float e = s - target;
      dy = e / B;
      l = 0.5f * e * e / B;
    }
    sm.dy[tid] = dy;
    A.dy[b0 + tid] = dy;
#pragma unroll
    for (int o = T_ROWS / 2; o > 0; o >>= 1) l += __shfl_xor_sync((1u << T_ROWS) - 1u, l, o);
    if (tid == 0) atomicAdd(loss, l);
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < T_U; ++j) {
    const int u = u0 + T_US * j;
    float v[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) v[r] = z2[j][r] > 0.f ? sm.dy[r0 + r] * w3[j] : 0.f;
    *reinterpret_cast<float4*>(&sm.d2[u][r0]) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(A.dZ2 + (size_t)u * A.ld + b0 + r0) = make_float4(v[0], v[1], v[2], v[3]);
  }
  __syncthreads();
  dot_rows<LH, LH + 4, false>(&sm.d2[0][r0], &sm.W.W2[0][u0], d);
#pragma unroll
  for (int j = 0; j < T_U; ++j) {
#pragma unroll
    for (int r = 0; r < 4; ++r) d[j][r] = z1[j][r] > 0.f ? d[j][r] : 0.f;
    *reinterpret_cast<float4*>(A.dZ1 + (size_t)(u0 + T_US * j) * A.ld + b0 + r0) =
        make_float4(d[j][0], d[j][1], d[j][2], d[j][3]);
  }
}

struct AdamArgs {
  float *p, *m, *v;  // parameters and moments
  float lr, b1, b2, eps, c1, c2;
};

// dW[o][i] = sum_b dZ[o][b] * A[i][b], db[o] = sum_b dZ[o][b]: a block makes
// 16 x 8 sums of a layer (the last layer: one row of 8) on two warps, two sums
// a thread, and the biases beside the first 8 inputs on a third.  kAdam: the
// step of Adam on each sum instead of writing it to g, its parameter and
// moments loaded before the sums.
// Every sum is a chain of B dependent FMAs (4 cycles each, 2 us at B = 1024),
// so all 20865 run on the chip at once (176 blocks).  Bound by the words read
// from shared memory (3 a row and warp) and one warp's issue rate: 8.4 cycles a
// row.  One sum a thread on four warps and four on one warp took 12-13, as
// did loading only 4 rows ahead.  The copies of T_STAGES chunks of T_CB rows
// are in flight together.
constexpr int T_TO = 16, T_TI = 8;    // units x inputs a block
constexpr int T_CB = 256;             // rows of the batch a chunk
constexpr int T_STAGES = 4;
constexpr int T_W_THREADS = 96;
struct TrainWgradSmem {  // rows padded by 16 bytes: 8 rows' 16-byte pieces in different banks
  float r[T_STAGES][T_TO + T_TI][T_CB + 4];  // the units' dz, then the inputs' a
  float past[16];                            // the inner loop's last load runs past its row
};
constexpr int T_W2_TILES = (LH / T_TO) * (LH / T_TI), T_W1_TILES = (LH / T_TO) * (LF / T_TI), T_W3_TILES = LH / T_TI;
constexpr int T_WGRAD_GRID = T_W2_TILES + T_W1_TILES + T_W3_TILES;

constexpr int L_OFF_W1 = 0;  // the parameter vector: W1 [LH][LF], b1 [LH], W2 [LH][LH], b2 [LH], w3 [LH], b3 [1]
constexpr int L_OFF_B1 = L_OFF_W1 + LH * LF;
constexpr int L_OFF_W2 = L_OFF_B1 + LH;
constexpr int L_OFF_B2 = L_OFF_W2 + LH * LH;
constexpr int L_OFF_W3 = L_OFF_B2 + LH;
constexpr int L_OFF_B3 = L_OFF_W3 + LH;
constexpr int L_NPARAM = L_OFF_B3 + 1;

struct AdamState {
  float p, m, v;
};
__device__ __forceinline__ AdamState adam_load(const AdamArgs& ad, int e) { return {ad.p[e], ad.m[e], ad.v[e]}; }
__device__ __forceinline__ float adam_step(const AdamArgs& ad, int e, AdamState a, float s) {
  a.m = fmaf(1.f - ad.b1, s, ad.b1 * a.m);
  a.v = fmaf((1.f - ad.b2) * s, s, ad.b2 * a.v);
  a.p -= ad.lr * (a.m / ad.c1) / (sqrtf(a.v / ad.c2) + ad.eps);
  ad.m[e] = a.m;
  ad.v[e] = a.v;
  ad.p[e] = a.p;
  return a.p;
}

template <bool kAdam>
__global__ void __launch_bounds__(T_W_THREADS) k_t_wgrad(TrainActs A, float* g, AdamArgs ad) {
  extern __shared__ __align__(16) unsigned char t_raw[];
  TrainWgradSmem& sm = *reinterpret_cast<TrainWgradSmem*>(t_raw);
  const int tid = threadIdx.x, lane = tid & 31;
  // this block's tile: units o0 .. o0 + no - 1 of dz, inputs i0 .. i0 + 7 of a
  int tile = blockIdx.x, I, offw, offb, no = T_TO, layer;
  const float *dz, *a;
  if (tile < T_W2_TILES) {
    layer = 2, I = LH, offw = L_OFF_W2, offb = L_OFF_B2, dz = A.dZ2, a = A.H1;
  } else if (tile < T_W2_TILES + T_W1_TILES) {
    tile -= T_W2_TILES;
    layer = 1, I = LF, offw = L_OFF_W1, offb = L_OFF_B1, dz = A.dZ1, a = A.X;
  } else {
    tile -= T_W2_TILES + T_W1_TILES;
    layer = 3, I = LH, offw = L_OFF_W3, offb = L_OFF_B3, dz = A.dy, a = A.H2, no = 1;
  }
  const int i0 = tile % (I / T_TI) * T_TI, o0 = tile / (I / T_TI) * T_TO;
  const int nchunk = (A.ld + T_CB - 1) / T_CB;
  ptx::grid_dependents_launch();
  ptx::grid_dependency_wait();
  auto load = [&](int c) {  // chunk c's rows, zeros past ld
    if (c < nchunk && tid < T_CB / 4) {  // warps 0 and 1: a thread's 4 columns of each row of the tile
      const int b = c * T_CB + 4 * tid;
      const uint32_t n = b < A.ld ? 16u : 0u;
      float* dst = &sm.r[c % T_STAGES][0][4 * tid];
      const float* src = dz + (size_t)o0 * A.ld + (n ? b : 0);
      for (int r = 0; r < no; ++r) ptx::cp_async16_zfill(dst + r * (T_CB + 4), src + (size_t)r * A.ld, n);
      dst += T_TO * (T_CB + 4);
      src = a + (size_t)i0 * A.ld + (n ? b : 0);
#pragma unroll
      for (int r = 0; r < T_TI; ++r) ptx::cp_async16_zfill(dst + r * (T_CB + 4), src + (size_t)r * A.ld, n);
    }
    ptx::cp_async_commit();
  };
  for (int c = 0; c < T_STAGES - 1; ++c) load(c);
  // warps 0 and 1: units o, o + 8 and input i of each lane; warp 2: the bias of unit `lane`
  const bool bias = tid >= 64;
  const int o = bias ? min(lane, T_TO - 1) : lane >> 2, i = (lane & 3) + 4 * (tid >> 5 & 1);
  const bool on = bias ? lane < no && i0 == 0 : o < no, two = on && !bias && no > 1;
  const int e0 = bias ? offb + o0 + o : offw + (o0 + o) * I + i0 + i, e1 = e0 + 8 * I;  // the sums' parameters
  AdamState st0{}, st1{};
  if (kAdam && on) st0 = adam_load(ad, e0);
  if (kAdam && two) st1 = adam_load(ad, e1);
  float s0 = 0.f, s1 = 0.f;
  for (int c = 0; c < nchunk; ++c) {
    ptx::cp_async_wait<T_STAGES - 2>();
    __syncthreads();  // chunk c has landed, and nobody reads the stage that the next copy overwrites
    load(c + T_STAGES - 1);
    if (!on) continue;
    const int n = min(T_CB, A.ld - c * T_CB) / 4;  // a multiple of 4
    const float4* zr = reinterpret_cast<const float4*>(sm.r[c % T_STAGES][o]);
    // 16 rows are loaded while the 16 before them are summed (the last load
    // runs past the row and is not used)
    if (bias) {
      float4 z[2][4];
      auto fetch = [&](int b, int h) {
#pragma unroll
        for (int q = 0; q < 4; ++q) z[h][q] = zr[b + q];
      };
      auto add = [&](int h) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          s0 += z[h][q].x;
          s0 += z[h][q].y;
          s0 += z[h][q].z;
          s0 += z[h][q].w;
        }
      };
      fetch(0, 0);
#pragma unroll 1
      for (int b = 0; b < n; b += 8) {
        fetch(b + 4, 1);
        add(0);
        if (b + 4 >= n) break;
        fetch(b + 8, 0);
        add(1);
      }
      continue;
    }
    // (the last layer has one unit: s1 is not used)
    const float4* zr8 = reinterpret_cast<const float4*>(sm.r[c % T_STAGES][two ? o + 8 : o]);
    const float4* ar = reinterpret_cast<const float4*>(sm.r[c % T_STAGES][T_TO + i]);
    float4 z[2][4], y[2][4], v[2][4];
    auto fetch = [&](int b, int h) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        z[h][q] = zr[b + q];
        y[h][q] = zr8[b + q];
        v[h][q] = ar[b + q];
      }
    };
    auto add = [&](int h) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        s0 = fmaf(z[h][q].x, v[h][q].x, s0);
        s1 = fmaf(y[h][q].x, v[h][q].x, s1);
        s0 = fmaf(z[h][q].y, v[h][q].y, s0);
        s1 = fmaf(y[h][q].y, v[h][q].y, s1);
        s0 = fmaf(z[h][q].z, v[h][q].z, s0);
        s1 = fmaf(y[h][q].z, v[h][q].z, s1);
        s0 = fmaf(z[h][q].w, v[h][q].w, s0);
        s1 = fmaf(y[h][q].w, v[h][q].w, s1);
      }
    };
    fetch(0, 0);
#pragma unroll 1
    for (int b = 0; b < n; b += 8) {
      fetch(b + 4, 1);
      add(0);
      if (b + 4 >= n) break;
      fetch(b + 8, 0);
      add(1);
    }
  }
  auto finish = [&](int e, const AdamState& st, float s, int oo) {
    if (!kAdam) {
      g[e] = s;
      return;
    }
    const float w = adam_step(ad, e, st, s);
    if (!bias && layer == 2) A.W->W2[oo][i0 + i] = bf(w);
    else if (!bias && layer == 1) A.W->W1[oo][i0 + i] = bf(w);
  };
  if (on) finish(e0, st0, s0, o0 + o);
  if (two) finish(e1, st1, s1, o0 + o + 8);
}

}  // namespace vnm

// ---------------------------------------------------------------------------
// Host
// ---------------------------------------------------------------------------
using namespace vnm;

struct vnm_mlp {
  int device = 0;
  float* p = nullptr;  // [L_NPARAM] master weights
  float* g = nullptr;  // gradients
  float* m = nullptr;  // Adam moments
  float* v = nullptr;
  int steps = 0;
};

namespace vnm {

static MlpW mlp_view(const vnm_mlp* n) {
  MlpW w;
  w.W1 = n->p + L_OFF_W1;
  w.b1 = n->p + L_OFF_B1;
  w.W2 = n->p + L_OFF_W2;
  w.b2 = n->p + L_OFF_B2;
  w.w3 = n->p + L_OFF_W3;
  w.b3 = n->p + L_OFF_B3;
  return w;
}

static size_t mlp_smem() { return sizeof(MlpSmem) + 1024; }

// Arena bytes and storage of a step's activations (batches of B rows).
static int train_ld(int B) { return (B + 15) / 16 * 16; }
static size_t train_bytes(int B) {
  const size_t ld = (size_t)train_ld(B);
  return arena_bytes(ld * LF, 4) + 4 * arena_bytes(ld * LH, 4) + arena_bytes(ld, 4) + arena_bytes(1, sizeof(TrainW));
}
static vnm_status train_acts(vnm_ctx* ctx, const vnm_mlp* n, int B, TrainActs& A) {
  A.ld = train_ld(B);
  const size_t ld = (size_t)A.ld;
  A.X = arena_take<float>(ctx, ld * LF);
  A.H1 = arena_take<float>(ctx, ld * LH);
  A.H2 = arena_take<float>(ctx, ld * LH);
  A.dZ1 = arena_take<float>(ctx, ld * LH);
  A.dZ2 = arena_take<float>(ctx, ld * LH);
  A.dy = arena_take<float>(ctx, ld);
  A.W = arena_take<TrainW>(ctx, 1);
  if (!A.X || !A.H1 || !A.H2 || !A.dZ1 || !A.dZ2 || !A.dy || !A.W) return VNM_ERR_NOMEM;
  VNM_CUDA_TRY(cudaFuncSetAttribute(k_t_rows, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)sizeof(TrainRowsSmem)));
  VNM_CUDA_TRY(cudaFuncSetAttribute(k_t_wgrad<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)sizeof(TrainWgradSmem)));
  VNM_CUDA_TRY(cudaFuncSetAttribute(k_t_wgrad<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)sizeof(TrainWgradSmem)));
  VNM_LAUNCH(ctx, k_t_round, 84, 256, 0, n->p + L_OFF_W1, n->p + L_OFF_W2, A.W);
  return VNM_OK;
}

// Forward and backward of one batch (device X [B][LF], t [B]): the batch's
// loss is added to *d_loss (zeroed by the caller), and the gradient goes to
// n->g or, with `adam`, straight into a step of Adam.
static vnm_status mlp_grad(vnm_ctx* ctx, vnm_mlp* n, const float* X, const float* t, int B, const TrainActs& A,
                           float* d_loss, const AdamArgs* adam) {
  // each kernel may be set up while the one before it runs; its own wait for
  // that one (grid_dependency_wait) comes before its first access to memory
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.stream = ctx->stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cfg.gridDim = dim3(A.ld / T_ROWS);
  cfg.blockDim = dim3(T_THREADS);
  cfg.dynamicSmemBytes = sizeof(TrainRowsSmem);
  VNM_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_t_rows, X, t, B, mlp_view(n), A, d_loss));
  cfg.gridDim = dim3(T_WGRAD_GRID);
  cfg.blockDim = dim3(T_W_THREADS);
  cfg.dynamicSmemBytes = sizeof(TrainWgradSmem);
  VNM_CUDA_TRY(cudaLaunchKernelEx(&cfg, adam ? k_t_wgrad<true> : k_t_wgrad<false>, A, n->g,
                                  adam ? *adam : AdamArgs{}));
  ctx->launches += 2;
  return VNM_OK;
}

}  // namespace vnm

using namespace vnm;

extern "C" {

int vnm_mlp_param_count(void) { return L_NPARAM; }

vnm_status vnm_mlp_create(vnm_ctx* ctx, unsigned seed, vnm_mlp** out) {
  if (!ctx || !out) return VNM_ERR_ARG;
  *out = nullptr;
  VNM_CUDA_TRY(cudaSetDevice(ctx->device));
  std::vector<float> h(L_NPARAM, 0.f);
  unsigned s = seed * 747796405u + 2891336453u;
  auto rnd = [&]() {  // uniform (-1, 1), PCG-style hash
    s = s * 747796405u + 2891336453u;
    unsigned x = ((s >> ((s >> 28) + 4)) ^ s) * 277803737u;
    x = (x >> 22) ^ x;
    return (x >> 8) * (2.0f / 16777216.0f) - 1.0f;
  };
  const float a1 = sqrtf(6.0f / LF), a2 = sqrtf(6.0f / LH), a3 = sqrtf(3.0f / LH);
  for (int i = 0; i < LH * LF; ++i) h[L_OFF_W1 + i] = a1 * rnd();
  for (int i = 0; i < LH * LH; ++i) h[L_OFF_W2 + i] = a2 * rnd();
  for (int i = 0; i < LH; ++i) h[L_OFF_W3 + i] = a3 * rnd();
  vnm_mlp* n = new vnm_mlp();
  n->device = ctx->device;
  void* base = nullptr;
  if (cudaMalloc(&base, sizeof(float) * L_NPARAM * 4) != cudaSuccess) {
    delete n;
    return VNM_ERR_NOMEM;
  }
  n->p = static_cast<float*>(base);
  n->g = n->p + L_NPARAM;
  n->m = n->g + L_NPARAM;
  n->v = n->m + L_NPARAM;
  cudaMemset(base, 0, sizeof(float) * L_NPARAM * 4);
  cudaMemcpy(n->p, h.data(), sizeof(float) * L_NPARAM, cudaMemcpyHostToDevice);
  *out = n;
  return VNM_OK;
}

vnm_status vnm_mlp_free(vnm_mlp* n) {
  if (!n) return VNM_ERR_ARG;
  cudaSetDevice(n->device);
  cudaFree(n->p);
  delete n;
  return VNM_OK;
}

vnm_status vnm_mlp_get(const vnm_mlp* n, float* params) {
  if (!n || !params) return VNM_ERR_ARG;
  VNM_CUDA_TRY(cudaMemcpy(params, n->p, sizeof(float) * L_NPARAM, cudaMemcpyDeviceToHost));
  return VNM_OK;
}

vnm_status vnm_mlp_set(vnm_mlp* n, const float* params) {
  if (!n || !params) return VNM_ERR_ARG;
  VNM_CUDA_TRY(cudaMemcpy(n->p, params, sizeof(float) * L_NPARAM, cudaMemcpyHostToDevice));
  n->steps = 0;
  VNM_CUDA_TRY(cudaMemset(n->m, 0, sizeof(float) * L_NPARAM * 2));
  return VNM_OK;
}

vnm_status vnm_mlp_grad(vnm_ctx* ctx, vnm_mlp* n, const float* X, const float* t, int B, float* grads,
                        float* loss) {
  if (!ctx || !n || !X || !t || B <= 0 || !grads || !loss) return VNM_ERR_ARG;
  VNM_TRY(arena_reserve(ctx, arena_bytes((size_t)B * LF, 4) + arena_bytes(B, 4) + train_bytes(B) + 4096));
  VNM_TRY(pinned_reserve(ctx, 64));
  VNM_TRY(begin_call(ctx));
  const float *dX, *dt;
  VNM_TRY(stage_in(ctx, X, (size_t)B * LF, VNM_MEM_HOST, &dX));
  VNM_TRY(stage_in(ctx, t, (size_t)B, VNM_MEM_HOST, &dt));
  float* dl = arena_take<float>(ctx, 1);
  if (!dl) return VNM_ERR_NOMEM;
  TrainActs A;
  VNM_TRY(train_acts(ctx, n, B, A));
  VNM_CUDA_TRY(cudaMemsetAsync(dl, 0, sizeof(float), ctx->stream));
  VNM_TRY(mlp_grad(ctx, n, dX, dt, B, A, dl, nullptr));
  VNM_CUDA_TRY(cudaMemcpyAsync(grads, n->g, sizeof(float) * L_NPARAM, cudaMemcpyDeviceToHost, ctx->stream));
  VNM_CUDA_TRY(cudaMemcpyAsync(loss, dl, sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
  return end_call(ctx);
}

// Adam steps over a dataset (host X [n][LF], t [n]): `epochs` passes in
// mini-batches of B (the data order is fixed; shuffle on the host).
vnm_status vnm_mlp_train(vnm_ctx* ctx, vnm_mlp* net, const float* X, const float* t, int n, int B, int epochs,
                         float lr, float* final_loss) {
  if (!ctx || !net || !X || !t || n <= 0 || B <= 0 || epochs <= 0) return VNM_ERR_ARG;
  const int nb = n / B;
  if (nb == 0) return VNM_ERR_ARG;
  VNM_TRY(arena_reserve(ctx, arena_bytes((size_t)n * LF, 4) + arena_bytes(n, 4) + train_bytes(B) +
                                 arena_bytes(nb + 1, 4) + 8192));
  VNM_TRY(pinned_reserve(ctx, 64 + nb));
  VNM_TRY(begin_call(ctx));
  const float *dX, *dt;
  VNM_TRY(stage_in(ctx, X, (size_t)n * LF, VNM_MEM_HOST, &dX));
  VNM_TRY(stage_in(ctx, t, (size_t)n, VNM_MEM_HOST, &dt));
  float* losses = arena_take<float>(ctx, nb + 1);
  if (!losses) return VNM_ERR_NOMEM;
  TrainActs A;
  VNM_TRY(train_acts(ctx, net, B, A));
  AdamArgs ad{net->p, net->m, net->v, lr, 0.9f, 0.999f, 1e-8f, 0.f, 0.f};
  for (int e = 0; e < epochs; ++e) {
    VNM_CUDA_TRY(cudaMemsetAsync(losses, 0, sizeof(float) * nb, ctx->stream));
    for (int k = 0; k < nb; ++k) {
      net->steps++;
      ad.c1 = 1.f - powf(ad.b1, (float)net->steps);
      ad.c2 = 1.f - powf(ad.b2, (float)net->steps);
      VNM_TRY(mlp_grad(ctx, net, dX + (size_t)k * B * LF, dt + (size_t)k * B, B, A, losses + k, &ad));
    }
  }
  VNM_CUDA_TRY(cudaMemcpyAsync(ctx->h_pinned, losses, sizeof(float) * nb, cudaMemcpyDeviceToHost, ctx->stream));
  VNM_TRY(end_call(ctx));
  if (final_loss) {
    double s = 0;
    const float* l = reinterpret_cast<const float*>(ctx->h_pinned);
    for (int k = 0; k < nb; ++k) s += l[k];
    *final_loss = (float)(s / nb);
  }
  return VNM_OK;
}

}  // extern "C"

namespace vnm {

static int lgrid(const vnm_ctx* ctx, long long n, int nt = 256) {
  long long g = (n + nt - 1) / nt;
  const long long cap = (long long)ctx->num_sms * 8;
  if (g > cap) g = cap;
  return g < 1 ? 1 : (int)g;
}

// The kernel's shared-memory ceiling, set for the call's device.
template <bool kPlain>
static vnm_status mlp_launch_prep(size_t smem) {
  VNM_CUDA_TRY(cudaFuncSetAttribute(k_l_mlp<kPlain>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  return VNM_OK;
}

}  // namespace vnm

extern "C" {

vnm_status vnm_mlp_forward(vnm_ctx* ctx, const vnm_mlp* net, const float* X, int n, float* Y) {
  if (!ctx || !net || n < 0 || (n > 0 && (!X || !Y))) return VNM_ERR_ARG;
  if (n == 0) return VNM_OK;
  VNM_TRY(arena_reserve(ctx, arena_bytes((size_t)n * LF, 4) + arena_bytes(n, 4) + arena_bytes(1, 4) + 1024));
  VNM_TRY(pinned_reserve(ctx, 64));
  VNM_TRY(begin_call(ctx));
  const float* dX;
  VNM_TRY(stage_in(ctx, X, (size_t)n * LF, VNM_MEM_HOST, &dX));
  float* dY = arena_take<float>(ctx, n);
  int* err = arena_take<int>(ctx, 1);
  if (!dY || !err) return VNM_ERR_NOMEM;
  VNM_CUDA_TRY(cudaMemsetAsync(err, 0, sizeof(int), ctx->stream));
  const size_t smem = mlp_smem();
  VNM_TRY(mlp_launch_prep<true>(smem));
  LMat L{};
  const int tiles = (n + 127) / 128;
  const int grid = tiles < ctx->num_sms ? tiles : ctx->num_sms;
  VNM_CUDA_TRY(cudaEventRecord(ctx->ev_main0, ctx->stream));
  VNM_LAUNCH(ctx, k_l_mlp<true>, grid, ML_THREADS, smem, L, mlp_view(net), MlpTail{}, nullptr, nullptr, 0, 0, 0u,
             nullptr, dX, n, dY, err);
  VNM_CUDA_TRY(cudaEventRecord(ctx->ev_main1, ctx->stream));
  VNM_CUDA_TRY(cudaMemcpyAsync(Y, dY, sizeof(float) * n, cudaMemcpyDeviceToHost, ctx->stream));
  VNM_CUDA_TRY(cudaMemcpyAsync(ctx->h_pinned, err, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  VNM_TRY(end_call(ctx));
  VNM_CUDA_TRY(cudaEventElapsedTime(&ctx->main_ms, ctx->ev_main0, ctx->ev_main1));
  return ctx->h_pinned[0] ? VNM_ERR_INTERNAL : VNM_OK;
}

vnm_status vnm_nm_learned(vnm_ctx* ctx, int nrows, int nnz, const int* row, const int* col, const float* val,
                          int mem, int N, int M, const vnm_mlp* net, const vnm_learned_params* prm,
                          vnm_learned_result* out, int* newpos) {
  if (!ctx || !prm || !out) return VNM_ERR_ARG;
  if (M < 2 || M > 8 || N < 1 || N >= M) return VNM_ERR_ARG;
  if (nrows < 0 || nnz < 0 || (nrows % M) != 0) return VNM_ERR_ARG;
  if (mem != VNM_MEM_HOST && mem != VNM_MEM_DEVICE) return VNM_ERR_ARG;
  if (nnz > 0 && (!row || !col || !val)) return VNM_ERR_ARG;
  if (nrows >= (1 << 27)) return VNM_ERR_LIMIT;  // 16 nrows + 1 row groups fit an int
  const int mode = prm->mode, KT = prm->targets;
  if (mode < VNM_LEARNED_MLP || mode > VNM_LEARNED_RANDOM) return VNM_ERR_ARG;
  if (mode == VNM_LEARNED_MLP && !net) return VNM_ERR_ARG;
  if (net && net->device != ctx->device) return VNM_ERR_ARG;
  if (prm->objective < 0 || prm->objective > 1 || prm->max_rounds < 0 || prm->patience < 1) return VNM_ERR_ARG;
  if (KT < 1 || KT * M * M > 2048) return VNM_ERR_ARG;
  if (mode != VNM_LEARNED_EXHAUSTIVE && (prm->topk < 1 || prm->topk > LTOP)) return VNM_ERR_ARG;
  if (prm->dump_cap < 0 || (prm->dump_cap > 0 && (!prm->dump_features || !prm->dump_gains))) return VNM_ERR_ARG;
  memset(out, 0, sizeof(*out));
  const int R = nrows, nseg = R / M;
  const long long gbytes = ((long long)R * nseg + 3) & ~3ll;
  const int dcap = prm->dump_every > 0 ? prm->dump_cap : 0;
  // chunks that columns, each in the list once at most, can have
  const size_t chunk_cap = (size_t)R + (size_t)nnz / L_CHUNK + 1;
  size_t need = pattern_bytes(R, nnz) + 3 * arena_bytes(nnz, 4) + arena_bytes(gbytes, 1) +
                arena_bytes((size_t)nseg * 9, 4) + arena_bytes(nseg, 4) + arena_bytes((size_t)R * 9, 4) +
                3 * arena_bytes(R + 1, 4) + 2 * arena_bytes(nseg + 1, 4) + arena_bytes((size_t)nseg * LTOP, 4) +
                2 * arena_bytes(nseg + 1, 8) + arena_bytes(nseg + 1, 16) + arena_bytes(nseg + 1, 8) +
                arena_bytes(LC_N + 8 * 2, 4) + 2 * arena_bytes(chunk_cap, 8) +
                arena_bytes((size_t)dcap * LF, 4) + arena_bytes(dcap, 4) + 8192;
  VNM_TRY(arena_reserve(ctx, need));
  VNM_TRY(pinned_reserve(ctx, 512));
  VNM_TRY(begin_call(ctx));
  const int *d_row, *d_col;
  const float* d_val;
  VNM_TRY(stage_in(ctx, row, nnz, mem, &d_row));
  VNM_TRY(stage_in(ctx, col, nnz, mem, &d_col));
  VNM_TRY(stage_in(ctx, val, nnz, mem, &d_val));
  Pattern P;
  VNM_TRY(build_pattern(ctx, R, nnz, d_row, d_col, d_val, N, M, P, ctx->h_pinned, false, false));
  LMat L;
  L.R = R;
  L.M = M;
  L.N = N;
  L.nseg = nseg;
  L.obj = prm->objective;
  L.cptr = P.cptr;
  L.crow = P.crow;
  L.G = arena_take<unsigned char>(ctx, gbytes > 0 ? gbytes : 4);
  L.hist = arena_take<int>(ctx, (size_t)nseg * 9 + 1);
  L.cnt = arena_take<int>(ctx, nseg + 1);
  L.colh = arena_take<int>(ctx, (size_t)R * 9 + 1);
  L.orig = arena_take<int>(ctx, R + 1);
  L.pos = arena_take<int>(ctx, R + 1);
  int* active = arena_take<int>(ctx, nseg + 1);
  int* top = arena_take<int>(ctx, (size_t)nseg * LTOP + 1);
  unsigned long long* best = arena_take<unsigned long long>(ctx, nseg + 1);
  unsigned long long* claim = arena_take<unsigned long long>(ctx, nseg + 1);
  int4* acc = arena_take<int4>(ctx, nseg + 1);
  int2* uw = arena_take<int2>(ctx, nseg + 1);            // the two nodes of each accepted swap
  int2* swap_items = arena_take<int2>(ctx, chunk_cap);  // chunks of accepted swaps' columns
  int2* col_items = arena_take<int2>(ctx, chunk_cap);   // chunks of columns to be counted
  // sums (cu: [0] gain [1] scored [2..3] totals) and counters, read back in one copy
  unsigned long long* cu = arena_take<unsigned long long>(ctx, 8 + LC_N / 2);
  int* ci = reinterpret_cast<int*>(cu + 8);
  float* dx = dcap ? arena_take<float>(ctx, (size_t)dcap * LF) : nullptr;
  float* dy = dcap ? arena_take<float>(ctx, dcap) : nullptr;
  int* d_newpos = arena_take<int>(ctx, R + 1);
  if (!L.G || !L.hist || !L.cnt || !L.colh || !L.orig || !L.pos || !active || !top || !best || !claim ||
      !acc || !uw || !swap_items || !col_items || !cu || !d_newpos || (dcap && (!dx || !dy)))
    return VNM_ERR_NOMEM;
  cudaStream_t st = ctx->stream;
  VNM_CUDA_TRY(cudaMemsetAsync(L.G, 0, gbytes > 0 ? gbytes : 4, st));
  VNM_CUDA_TRY(cudaMemsetAsync(cu, 0, 8 * sizeof(unsigned long long) + LC_N * sizeof(int), st));
  if (R > 0) VNM_LAUNCH(ctx, k_l_iota2, lgrid(ctx, R), 256, 0, L.orig, L.pos, R);
  if (P.np > 0)
    VNM_LAUNCH(ctx, k_l_build_G, lgrid(ctx, nnz), 256, 0, d_row, d_col, d_val, nnz, M, nseg,
               reinterpret_cast<unsigned*>(L.G));
  if (nseg > 0) {
    VNM_LAUNCH(ctx, k_l_all_columns, lgrid(ctx, R), 256, 0, L, col_items, ci + LC_COL_ITEMS);
    VNM_LAUNCH(ctx, k_l_colh_rows, lgrid(ctx, (long long)R * 32), 256, 0, L, col_items, ci + LC_COL_ITEMS);
    VNM_LAUNCH(ctx, k_l_seg_hist, lgrid(ctx, nseg), 256, 0, L);
    VNM_LAUNCH(ctx, k_l_totals, lgrid(ctx, nseg), 256, 0, L.hist, nseg, N, cu + 2);
  }
  unsigned long long* hcu = reinterpret_cast<unsigned long long*>(ctx->h_pinned);  // 8 words
  int* hci = reinterpret_cast<int*>(hcu + 8);                                       // LC_N ints, as on the device
  VNM_CUDA_TRY(cudaMemcpyAsync(hcu, cu, sizeof(unsigned long long) * 4, cudaMemcpyDeviceToHost, st));
  float* hb = reinterpret_cast<float*>(ctx->h_pinned + 64);
  if (mode == VNM_LEARNED_MLP) {
    VNM_CUDA_TRY(cudaMemcpyAsync(hb, net->p + L_OFF_B1, sizeof(float) * LH, cudaMemcpyDeviceToHost, st));
    VNM_CUDA_TRY(cudaMemcpyAsync(hb + LH, net->p + L_OFF_B2, sizeof(float) * (2 * LH + 1), cudaMemcpyDeviceToHost, st));
  }
  VNM_CUDA_TRY(cudaStreamSynchronize(st));
  MlpTail T{};
  static_assert(sizeof(T) == sizeof(float) * (3 * LH + 1), "the tail as copied");
  if (mode == VNM_LEARNED_MLP) memcpy(&T, hb, sizeof(T));
  out->init_invalid = out->final_invalid = (long long)hcu[2];
  out->init_retained = out->final_retained = (long long)hcu[3];
  const size_t smem = mlp_smem();
  if (mode == VNM_LEARNED_MLP) VNM_TRY(mlp_launch_prep<false>(smem));
  const MlpW W = net ? mlp_view(net) : MlpW{};
  const int pgrid = ctx->num_sms;  // the blocks beyond the active segments return at once
  const int egrid = ctx->num_sms * 8;
  const size_t state_bytes = 8 * sizeof(unsigned long long) + LC_N * sizeof(int);
  int idle = 0, rounds = 0, swaps = 0;
  VNM_CUDA_TRY(cudaEventRecord(ctx->ev_main0, st));
  for (int round = 0; round < prm->max_rounds && nseg >= 2 && P.np > 0; ++round) {
    VNM_LAUNCH(ctx, k_l_round_start, 1 + lgrid(ctx, nseg, L_START_THREADS), L_START_THREADS, 0, L, active, ci, best,
               claim);
    if (mode == VNM_LEARNED_MLP)
      VNM_LAUNCH(ctx, k_l_mlp<false>, pgrid, ML_THREADS, smem, L, W, T, active, ci + LC_ACTIVE, KT, round,
                 prm->seed, top, nullptr, 0, nullptr, ci + LC_ERR);
    VNM_LAUNCH(ctx, k_l_exact, egrid, 256, 0, L, active, ci, KT, round, prm->seed, top, mode, prm->topk, best, dx, dy,
               prm->dump_every, ci + LC_DUMP, dcap, cu + 1);
    VNM_LAUNCH(ctx, k_l_claim, lgrid(ctx, nseg), 256, 0, L, active, ci, round, prm->seed, best, claim);
    VNM_LAUNCH(ctx, k_l_accept, lgrid(ctx, nseg), 256, 0, L, active, ci, round, prm->seed, best, claim, acc, uw,
               swap_items, cu);
    VNM_LAUNCH(ctx, k_l_apply_rows, egrid, 256, 0, L, acc, ci, uw, swap_items, col_items);
    VNM_LAUNCH(ctx, k_l_colh_rows, egrid, 256, 0, L, col_items, ci + LC_COL_ITEMS);
    VNM_CUDA_TRY(cudaMemcpyAsync(hcu, cu, state_bytes, cudaMemcpyDeviceToHost, st));
    VNM_CUDA_TRY(cudaStreamSynchronize(st));
    if (hci[LC_ERR]) return VNM_ERR_INTERNAL;
    rounds = round + 1;
    if (hci[LC_ACTIVE] == 0) break;  // no segment holds an invalid group
    swaps += hci[LC_ACC];
    idle = hci[LC_ACC] == 0 ? idle + 1 : 0;
    if (idle >= prm->patience) break;
    if (prm->stop_gain > 0 && (long long)hcu[0] >= prm->stop_gain) break;
  }
  VNM_CUDA_TRY(cudaEventRecord(ctx->ev_main1, st));
  VNM_CUDA_TRY(cudaMemsetAsync(cu + 2, 0, sizeof(unsigned long long) * 2, st));
  if (nseg > 0) VNM_LAUNCH(ctx, k_l_totals, lgrid(ctx, nseg), 256, 0, L.hist, nseg, N, cu + 2);
  VNM_CUDA_TRY(cudaMemcpyAsync(hcu, cu, state_bytes, cudaMemcpyDeviceToHost, st));
  VNM_CUDA_TRY(cudaStreamSynchronize(st));
  VNM_CUDA_TRY(cudaEventElapsedTime(&ctx->main_ms, ctx->ev_main0, ctx->ev_main1));
  out->final_invalid = (long long)hcu[2];
  out->final_retained = (long long)hcu[3];
  out->gain = (long long)hcu[0];
  out->exact_scored = (long long)hcu[1];
  out->rounds = rounds;
  out->swaps = swaps;
  out->ndump = hci[LC_DUMP] < dcap ? hci[LC_DUMP] : dcap;
  for (int q = 0; q < 28; ++q) ctx->stats[q] = 0;
  ctx->stats[0] = rounds;
  ctx->stats[1] = out->exact_scored;
  ctx->stats[2] = swaps;
  ctx->stats[3] = nseg;
  ctx->stats[5] = P.np;
  if (out->ndump) {
    VNM_CUDA_TRY(cudaMemcpyAsync(prm->dump_features, dx, sizeof(float) * LF * out->ndump, cudaMemcpyDeviceToHost, st));
    VNM_CUDA_TRY(cudaMemcpyAsync(prm->dump_gains, dy, sizeof(float) * out->ndump, cudaMemcpyDeviceToHost, st));
  }
  if (newpos && R > 0) {
    VNM_LAUNCH(ctx, k_l_invert, lgrid(ctx, R), 256, 0, L.orig, R, d_newpos);
    VNM_CUDA_TRY(cudaMemcpyAsync(newpos, d_newpos, sizeof(int) * R, cudaMemcpyDeviceToHost, st));
  }
  return end_call(ctx);
}

}  // extern "C"
