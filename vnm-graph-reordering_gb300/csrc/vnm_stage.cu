// VNM stage on the GPU: the row sort of reordering.py, rebuilt.
//
// The reference runs this stage as a Python subprocess (main.cu:116-153) over
// strings: it builds an M-character bit string per (row, segment)
// (generate_segmat, reordering.py:113-119), hashes each to its index in the
// reflected Gray code, negated when it has more than two ones
// (construct_bitcode_hash_tab, :95-107), stable-sorts the rows by the tuple
// of their hashes (:219), maps row -> new_id[row] and col -> new_id[col]
// with new_id[i] = sorted[i] (:223-229, :171-177), recounts the V-blocks
// whose OR has more than four ones (and, strictly, blocks with a row of more
// than two ones) (:125-152), and stops when the count grows (:242-246).
//
// Here every round is a handful of kernels over the COO:
//   1. radix-sort the entries by (row, col)                       -> groups
//   2. group bits, Gray-code hash, one sortable token per group
//   3. V-block counts with a dense OR table (blocks x segments bytes)
//   4. the row order: rows compared as token strings, ties kept in index
//      order.  Done by refinement: sort rows by (group of the previous
//      pass, k-th token) with the stable radix sort until no group of equal
//      rows can still be split.
// For m <= 65536 rows and nseg <= 16384 segments nothing is sorted by entry
// and a round is four kernels: the entries stay in the original matrix's rows
// (a round only composes the node map), one warp per row turns its columns
// into the token list (k_vs_tokens), and one thread-block cluster holds all
// rows in its shared memory and refines their order there (k_vs_order).
// Token order: comparing the dense hash tuples of two rows is the same as
// comparing their lists of (segment, hash) tokens, where token (s, h) ranks
// by  h > 0: +(nseg - s),  h < 0: -(nseg - s),  end of row: 0, then by h.
#include <cooperative_groups.h>

#include <cstdlib>
#include <cstring>
#include <vector>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace vnm {

constexpr int VS_NT = 256;

static inline int vs_grid(const vnm_ctx* ctx, long long n) {
  long long g = (n + VS_NT - 1) / VS_NT, cap = (long long)ctx->num_sms * 16;
  if (g > cap) g = cap;
  return g < 1 ? 1 : (int)g;
}

static inline int bits_for(long long v) {  // bits to hold 0..v
  int b = 1;
  while ((1ll << b) <= v) ++b;
  return b;
}

__global__ void k_vs_keys(const int* row, const int* col, int nnz, int colbits, unsigned long long* keys) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nnz; i += gridDim.x * blockDim.x)
    keys[i] = ((unsigned long long)(unsigned)row[i] << colbits) | (unsigned)col[i];
}

// group heads among (row, col)-sorted keys: a new (row, col / M) pair
__global__ void k_vs_heads(const unsigned long long* keys, int nnz, int colbits, int M, int* flag) {
  const unsigned long long cmask = (1ull << colbits) - 1;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nnz; i += gridDim.x * blockDim.x) {
    const unsigned long long k = keys[i];
    int f = 1;
    if (i > 0) {
      const unsigned long long p = keys[i - 1];
      f = ((p >> colbits) != (k >> colbits)) || ((int)(p & cmask) / M != (int)(k & cmask) / M);
    }
    flag[i] = f;
  }
}

__device__ __forceinline__ int gray_rank(unsigned code) {  // index of `code` in the reflected Gray code list
  unsigned idx = code;
  idx ^= idx >> 1;
  idx ^= idx >> 2;
  idx ^= idx >> 4;
  idx ^= idx >> 8;
  return (int)idx;
}

// One group per head: bits (offset k at bit M-1-k, as int(segmat, 2)),
// the token, and the row.  Also the V-block OR table and the strict flags.
__global__ void k_vs_groups(const unsigned long long* keys, const int* gpos, int nnz, int colbits, int M, int nseg,
                            int V, int* grow, int* gseg, unsigned* gtok, unsigned* ortab, unsigned* badtab) {
  const unsigned long long cmask = (1ull << colbits) - 1;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nnz; i += gridDim.x * blockDim.x) {
    const unsigned long long k = keys[i];
    const int r = (int)(k >> colbits), c = (int)(k & cmask), s = c / M;
    if (i > 0) {
      const unsigned long long p = keys[i - 1];
      if ((int)(p >> colbits) == r && (int)(p & cmask) / M == s) continue;  // not a head
    }
    unsigned bits = 0;
    for (int q = 0; q < M && i + q < nnz; ++q) {
      const unsigned long long kk = keys[i + q];
      if ((int)(kk >> colbits) != r || (int)(kk & cmask) / M != s) break;
      bits |= 1u << (M - 1 - (int)(kk & cmask) % M);
    }
    const int pc = __popc(bits);
    const int g = gpos[i];
    const int h = pc <= 2 ? gray_rank(bits) : -gray_rank(bits);
    const int rank = h > 0 ? (nseg - s) : -(nseg - s);
    grow[g] = r;
    gseg[g] = s;
    gtok[g] = ((unsigned)(rank + nseg) << 9) | (unsigned)(h + 256);
    const long long cell = (long long)(r / V) * nseg + s;
    atomicOr(&ortab[cell >> 2], bits << ((cell & 3) * 8));
    if (pc > 2) atomicOr(&badtab[cell >> 2], 1u << ((cell & 3) * 8));
  }
}

// kClear: the tables are left zero for the next round.  (A constant: with
// stores that might follow, the loads of the next words wait, 336 us instead of
// 269 over the 2 x 312 MB of 400000 rows at V = 64.)
template <bool kClear>
__global__ void k_vs_count(unsigned* ortab, unsigned* badtab, long long ncells, int* out2) {
  int inv = 0, strict = 0;
  for (long long w = blockIdx.x * (long long)blockDim.x + threadIdx.x; w < (ncells + 3) / 4;
       w += (long long)gridDim.x * blockDim.x) {
    const unsigned o = ortab[w], b = badtab[w];
    if (kClear && o) ortab[w] = 0u;
    if (kClear && b) badtab[w] = 0u;
    for (int q = 0; q < 4; ++q) {
      if (w * 4 + q >= ncells) break;
      const unsigned ob = (o >> (8 * q)) & 0xffu;
      const bool a = __popc(ob) > 4;
      inv += a;
      strict += a || ((b >> (8 * q)) & 0xffu);
    }
  }
  __shared__ int sum[2];
  if (threadIdx.x < 2) sum[threadIdx.x] = 0;
  __syncthreads();
  inv = __reduce_add_sync(0xffffffffu, inv);
  strict = __reduce_add_sync(0xffffffffu, strict);
  if ((threadIdx.x & 31) == 0 && strict) {  // (an invalid block is also a strictly invalid one)
    atomicAdd(&sum[0], inv);
    atomicAdd(&sum[1], strict);
  }
  __syncthreads();
  if (threadIdx.x < 2 && sum[threadIdx.x]) atomicAdd(&out2[threadIdx.x], sum[threadIdx.x]);
}

// first group of each row (groups are sorted by row)
__global__ void k_vs_rowptr(const int* grow, int ng, int m, int* rowptr) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r <= m; r += gridDim.x * blockDim.x) {
    int lo = 0, hi = ng;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (grow[mid] < r) lo = mid + 1;
      else hi = mid;
    }
    rowptr[r] = lo;
  }
}

__global__ void k_vs_iota(int* a, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) a[i] = i;
}

// keys for refinement pass k over rows in the current order:
// (group start << tokbits) | token_k ; rows that are settled keep token 0
__global__ void k_vs_refine_keys(const int* order, const int* gstart, const unsigned char* settled,
                                 const int* rowptr, const unsigned* gtok, int m, int k, int nseg, int tokbits,
                                 unsigned long long* keys, int* active) {
  const unsigned endtok = ((unsigned)nseg << 9) | 256u;
  int act = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
    const int r = order[i];
    unsigned tok = 0;
    if (!settled[i]) {
      const int g = rowptr[r] + k;
      tok = g < rowptr[r + 1] ? gtok[g] : endtok;
      act = 1;
    }
    keys[i] = ((unsigned long long)(unsigned)gstart[i] << tokbits) | tok;
  }
  if (__syncthreads_or(act) && threadIdx.x == 0) atomicOr(active, 1);
}

// after sorting by (group start, token): new group starts and settled flags.
// A row is settled when it is alone in its new group, or its token was the
// end of its row (all rows of the group are then equal).
__global__ void k_vs_regroup(const unsigned long long* skeys, const int* spos, const int* old_order, int m,
                             int tokbits, int nseg, int* new_order, int* head) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
    new_order[i] = old_order[spos[i]];
    head[i] = (i == 0 || skeys[i] != skeys[i - 1]) ? i : 0;
  }
}

__global__ void k_vs_settle(const unsigned long long* skeys, const int* gstart_new, int m, int tokbits, int nseg,
                            unsigned char* settled) {
  const unsigned endtok = ((unsigned)nseg << 9) | 256u;
  const unsigned long long tmask = (1ull << tokbits) - 1;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
    const int g = gstart_new[i];
    const bool alone = (i == g) && (i + 1 == m || gstart_new[i + 1] != g);
    const unsigned tok = (unsigned)(skeys[i] & tmask);
    settled[i] = alone || tok == endtok || tok == 0u;
  }
}

// inclusive max-scan of head positions -> group start of every position
__global__ void k_vs_maxscan_block(int* a, int n, int* blockmax) {
  __shared__ int s[1024];
  const int i = blockIdx.x * 1024 + threadIdx.x;
  int v = i < n ? a[i] : 0;
  s[threadIdx.x] = v;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {
    int t = threadIdx.x >= o ? s[threadIdx.x - o] : 0;
    __syncthreads();
    if (t > s[threadIdx.x]) s[threadIdx.x] = t;
    __syncthreads();
  }
  if (i < n) a[i] = s[threadIdx.x];
  if (threadIdx.x == 1023) blockmax[blockIdx.x] = s[1023];
}

__global__ void k_vs_maxscan_fix(int* a, int n, const int* blockmax) {
  const int b = blockIdx.x;
  if (b == 0) return;
  int carry = 0;
  for (int q = 0; q < b; ++q) carry = max(carry, blockmax[q]);
  const int i = b * 1024 + threadIdx.x;
  if (i < n && a[i] < carry) a[i] = carry;
}

__global__ void k_vs_apply(int* row, int* col, int nnz, const int* new_id) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nnz; i += gridDim.x * blockDim.x) {
    row[i] = new_id[row[i]];
    col[i] = new_id[col[i]];
  }
}

__global__ void k_vs_compose(int* comp, int m, const int* new_id) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) comp[i] = new_id[comp[i]];
}

struct VnmWork {
  int m, nnz, M, V, nseg, nblk, colbits, tokbits;
  long long ncells;
  // arena buffers
  unsigned long long* keys;
  int* flag;
  int* grow;
  int* gseg;
  unsigned* gtok;
  int* rowptr;
  unsigned* ortab;
  unsigned* badtab;
  int* counts;   // [2]
  int* order;    // [m]
  int* order2;   // [m]
  int* gstart;   // [m]
  unsigned char* settled;
  unsigned long long* rkeys;
  int* active;
  int* blockmax;
  int ng;
};

// Groups, tokens and counts of the current matrix (row, col) -> W.counts.
static vnm_status vnm_analyse(vnm_ctx* ctx, const int* row, const int* col, VnmWork& W, int* h2) {
  const int nnz = W.nnz;
  const size_t mark = ctx->arena.used;  // sort buffers are released at the end
  VNM_CUDA_TRY(cudaMemsetAsync(W.counts, 0, 2 * sizeof(int), ctx->stream));
  VNM_CUDA_TRY(cudaMemsetAsync(W.ortab, 0, ((W.ncells + 3) / 4) * 4, ctx->stream));
  VNM_CUDA_TRY(cudaMemsetAsync(W.badtab, 0, ((W.ncells + 3) / 4) * 4, ctx->stream));
  W.ng = 0;
  if (nnz > 0) {
    VNM_LAUNCH(ctx, k_vs_keys, vs_grid(ctx, nnz), VS_NT, 0, row, col, nnz, W.colbits, W.keys);
    unsigned long long* sk;
    int* sv;
    VNM_TRY(radix_sort_u64(ctx, W.keys, nullptr, nnz, 2 * W.colbits, &sk, &sv));
    VNM_LAUNCH(ctx, k_vs_heads, vs_grid(ctx, nnz), VS_NT, 0, sk, nnz, W.colbits, W.M, W.flag);
    int* d_ng = arena_take<int>(ctx, 1);
    if (!d_ng) return VNM_ERR_NOMEM;
    VNM_TRY(exclusive_scan(ctx, W.flag, W.flag, nnz, d_ng));
    VNM_LAUNCH(ctx, k_vs_groups, vs_grid(ctx, nnz), VS_NT, 0, sk, W.flag, nnz, W.colbits, W.M, W.nseg, W.V, W.grow,
               W.gseg, W.gtok, W.ortab, W.badtab);
    VNM_CUDA_TRY(cudaMemcpyAsync(h2 + 2, d_ng, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  }
  VNM_LAUNCH(ctx, k_vs_count<false>, vs_grid(ctx, (W.ncells + 3) / 4), VS_NT, 0, W.ortab, W.badtab, W.ncells, W.counts);
  VNM_CUDA_TRY(cudaMemcpyAsync(h2, W.counts, 2 * sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  VNM_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  if (nnz > 0) W.ng = h2[2];
  ctx->arena.used = mark;
  return VNM_OK;
}

static vnm_status maxscan(vnm_ctx* ctx, int* a, int n, int* blockmax) {
  const int nb = (n + 1023) / 1024;
  VNM_LAUNCH(ctx, k_vs_maxscan_block, nb, 1024, 0, a, n, blockmax);
  if (nb > 1) VNM_LAUNCH(ctx, k_vs_maxscan_fix, nb, 1024, 0, a, n, blockmax);
  return VNM_OK;
}

// The stable row order of reordering.py:219 for the analysed matrix.
static vnm_status vnm_row_order(vnm_ctx* ctx, VnmWork& W, int* h) {
  const int m = W.m;
  VNM_LAUNCH(ctx, k_vs_rowptr, vs_grid(ctx, m + 1), VS_NT, 0, W.grow, W.ng, m, W.rowptr);
  VNM_LAUNCH(ctx, k_vs_iota, vs_grid(ctx, m), VS_NT, 0, W.order, m);
  VNM_CUDA_TRY(cudaMemsetAsync(W.gstart, 0, sizeof(int) * m, ctx->stream));
  VNM_CUDA_TRY(cudaMemsetAsync(W.settled, 0, m, ctx->stream));
  const int keybits = W.tokbits + bits_for(m);
  for (int k = 0; k <= m; ++k) {  // at most one pass per token of the longest row
    VNM_CUDA_TRY(cudaMemsetAsync(W.active, 0, sizeof(int), ctx->stream));
    VNM_LAUNCH(ctx, k_vs_refine_keys, vs_grid(ctx, m), VS_NT, 0, W.order, W.gstart, W.settled, W.rowptr, W.gtok, m,
               k, W.nseg, W.tokbits, W.rkeys, W.active);
    VNM_CUDA_TRY(cudaMemcpyAsync(h, W.active, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    VNM_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    if (!h[0]) break;
    const size_t mark = ctx->arena.used;
    unsigned long long* sk;
    int* sp;
    VNM_TRY(radix_sort_u64(ctx, W.rkeys, nullptr, m, keybits, &sk, &sp));
    VNM_LAUNCH(ctx, k_vs_regroup, vs_grid(ctx, m), VS_NT, 0, sk, sp, W.order, m, W.tokbits, W.nseg, W.order2,
               W.gstart);
    VNM_TRY(maxscan(ctx, W.gstart, m, W.blockmax));
    VNM_LAUNCH(ctx, k_vs_settle, vs_grid(ctx, m), VS_NT, 0, sk, W.gstart, m, W.tokbits, W.nseg, W.settled);
    std::swap(W.order, W.order2);
    VNM_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    ctx->arena.used = mark;  // the sort's buffers are free again
  }
  return VNM_OK;
}

static size_t vnm_bytes(int m, int nnz, long long ncells) {
  size_t b = arena_bytes(nnz, 8) + arena_bytes(nnz, 4) * 3 + arena_bytes(nnz, 4) + arena_bytes(m + 1, 4);
  b += 2 * arena_bytes((ncells + 3) / 4, 4) + arena_bytes(2, 4);
  b += 4 * arena_bytes(m, 4) + arena_bytes(m, 1) + arena_bytes(m, 8) + arena_bytes(1, 4) +
       arena_bytes(m / 1024 + 2, 4);
  b += radix_sort_scratch_bytes(nnz > m ? nnz : m) + scan_scratch_bytes(nnz > 0 ? nnz : 1) + 4096;
  // per-round copies of the matrix and the composed map
  b += 4 * arena_bytes(nnz, 4) + 3 * arena_bytes(m, 4);
  return b;
}

static vnm_status vnm_setup(vnm_ctx* ctx, int m0, int n0, int nnz, int M, int V, VnmWork& W) {
  const int m = (m0 + M - 1) / M * M, n = (n0 + M - 1) / M * M;  // reordering.py:50-51
  W.m = m;
  W.nnz = nnz;
  W.M = M;
  W.V = V;
  W.nseg = n / M;
  W.nblk = (m + V - 1) / V;
  W.ncells = (long long)W.nblk * W.nseg;
  W.colbits = bits_for(n > m ? n : m);
  W.tokbits = bits_for(2ll * W.nseg) + 9;
  const int nn = nnz > 0 ? nnz : 1;
  W.keys = arena_take<unsigned long long>(ctx, nn);
  W.flag = arena_take<int>(ctx, nn);
  W.grow = arena_take<int>(ctx, nn);
  W.gseg = arena_take<int>(ctx, nn);
  W.gtok = arena_take<unsigned>(ctx, nn);
  W.rowptr = arena_take<int>(ctx, m + 1);
  W.ortab = arena_take<unsigned>(ctx, (W.ncells + 3) / 4);
  W.badtab = arena_take<unsigned>(ctx, (W.ncells + 3) / 4);
  W.counts = arena_take<int>(ctx, 2);
  W.order = arena_take<int>(ctx, m);
  W.order2 = arena_take<int>(ctx, m);
  W.gstart = arena_take<int>(ctx, m);
  W.settled = arena_take<unsigned char>(ctx, m);
  W.rkeys = arena_take<unsigned long long>(ctx, m);
  W.active = arena_take<int>(ctx, 1);
  W.blockmax = arena_take<int>(ctx, m / 1024 + 2);
  if (!W.keys || !W.flag || !W.grow || !W.gseg || !W.gtok || !W.rowptr || !W.ortab || !W.badtab || !W.counts ||
      !W.order || !W.order2 || !W.gstart || !W.settled || !W.rkeys || !W.active || !W.blockmax)
    return VNM_ERR_NOMEM;
  return VNM_OK;
}

__global__ void k_vs_check(const int* row, const int* col, int nnz, int m, int n, int* err) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nnz; i += gridDim.x * blockDim.x)
    if (row[i] < 0 || row[i] >= m || col[i] < 0 || col[i] >= n) atomicOr(err, 1);
}

static vnm_status vnm_args(vnm_ctx* ctx, int m, int n, int nnz, const int* row, const int* col, int mem, int M,
                           int V) {
  if (!ctx || m < 0 || n < 0 || nnz < 0 || M < 2 || M > 8 || V < 1) return VNM_ERR_ARG;
  if (mem != VNM_MEM_HOST && mem != VNM_MEM_DEVICE) return VNM_ERR_ARG;
  if (nnz > 0 && (!row || !col)) return VNM_ERR_ARG;
  if (m > (1 << 24) || n > (1 << 24)) return VNM_ERR_LIMIT;
  return VNM_OK;
}

// ---------------------------------------------------------------------------
// Rounds on the original rows
// ---------------------------------------------------------------------------
constexpr int VO_MAX_ROWS = 65536, VO_MAX_SEG = 16384;

// A token of the rows' order, in bits_for(2 nseg) + 8 bits and never 0:
// (rank + nseg) << 8, then h, or 256 + h of a negative one.
__device__ __forceinline__ unsigned vs_token(unsigned bits, int s, int nseg) {
  const int h = gray_rank(bits);
  return __popc(bits) <= 2 ? (unsigned)(2 * nseg - s) << 8 | (unsigned)h : (unsigned)s << 8 | (unsigned)(256 - h);
}

// Entries per row; lanes of a warp with the same row add once.
__global__ void k_vs_rowcount(const int* row, int nnz, int* count) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nnz; i += gridDim.x * blockDim.x) {
    const int r = row[i];
    const unsigned peers = __match_any_sync(__activemask(), r);
    if ((int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&count[r], __popc(peers));
  }
}

// Columns by row (any order inside a row; `fill` zero on entry).
__global__ void k_vs_rowfill(const int* row, const int* col, int nnz, const int* rowptr, int* fill, int* ccol) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nnz; i += gridDim.x * blockDim.x) {
    const int r = row[i], lane = threadIdx.x & 31;
    const unsigned peers = __match_any_sync(__activemask(), r);
    const int lead = __ffs(peers) - 1;
    int at = 0;
    if (lane == lead) at = atomicAdd(&fill[r], __popc(peers));
    at = __shfl_sync(peers, at, lead);
    ccol[rowptr[r] + at + __popc(peers & ((1u << lane) - 1u))] = col[i];
  }
}

// The composed map (identity without prev) and where its value lies:
// segment << 3 | place in the segment.
__global__ void k_vs_map(const int* prev, const int* new_id, int m, int M, int* comp, int* packed) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
    const int c = prev ? new_id[prev[i]] : i;
    comp[i] = c;
    packed[i] = (c / M) << 3 | (c % M);
  }
}

// Token list of every row, at the row's place in the column list, and the
// V-block tables; one warp a row.  A row of at most 32 entries is sorted in
// registers; a longer one sets its bits in a bitmap of one byte a segment in
// shared memory and reads the touched parts back in order; one of more than
// VT_LONG takes a block of its own, the first `nlb` blocks walking the list of
// those rows (on one warp a hub row's chain of gathers, and in one block the
// hubs that share their low bits, set the kernel's time: 27 us at 16384 rows,
// 262144 entries, 18 now).  Bound by the gathers of `packed` and the
// atomics of the tables.
constexpr int VT_WARPS = 8, VT_LONG = 128;
// The rows of more than VT_LONG entries; *n counts them (zero on entry).
__global__ void k_vs_long(const int* rowptr, int m, int* list, int* n) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < m; r += gridDim.x * blockDim.x)
    if (rowptr[r + 1] - rowptr[r] > VT_LONG) list[atomicAdd(n, 1)] = r;
}

__global__ void __launch_bounds__(VT_WARPS * 32)
    k_vs_tokens(const int* __restrict__ rowptr, const int* __restrict__ ccol, const int* __restrict__ comp,
                const int* __restrict__ packed, const int* __restrict__ longs, const int* __restrict__ nlong, int nlb,
                int m, int M, int nseg, int V, int2* tlist, unsigned* gtok, unsigned* ortab, unsigned* badtab) {
  extern __shared__ unsigned vt_bitmap[];
  __shared__ int wsum[VT_WARPS];
  const int nw = (nseg + 3) / 4;                     // words of a row's bitmap
  const int part = ((nw + 31) / 32 + 31) / 32 * 32;  // words a bit of the touched mask stands for
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned* bm = vt_bitmap + warp * nw;
  auto emit = [&](int b, long long cell0, int s, unsigned bits, int at) {
    gtok[b + at] = vs_token(bits, s, nseg);
    const long long cell = cell0 + s;
    atomicOr(&ortab[cell >> 2], bits << ((cell & 3) * 8));
    if (__popc(bits) > 2) atomicOr(&badtab[cell >> 2], 1u << ((cell & 3) * 8));
  };
  // entries first, first + step, ... of row b .. b + len into the bitmap t; the parts of it that were touched
  auto set_bits = [&](unsigned* t, int b, int len, int first, int step) {
    constexpr int U = 4;  // entries a lane in flight
    unsigned touched = 0;
    for (int e0 = first; e0 < len; e0 += step * U) {
      int c[U], p[U];
#pragma unroll
      for (int u = 0; u < U; ++u) c[u] = e0 + step * u < len ? ccol[b + e0 + step * u] : -1;
#pragma unroll
      for (int u = 0; u < U; ++u) p[u] = c[u] >= 0 ? packed[c[u]] : 0;
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (c[u] >= 0) {
          const int s = p[u] >> 3;
          atomicOr(&t[s >> 2], (1u << (M - 1 - (p[u] & 7))) << ((s & 3) * 8));
          touched |= 1u << ((s >> 2) / part);
        }
    }
    return touched;
  };
  auto nonzero_bytes = [](unsigned word) {
    int c = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) c += ((word >> (8 * k)) & 0xffu) ? 1 : 0;
    return c;
  };
  auto warp_incl = [&](int v) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += t;
    }
    return v;
  };
  if ((int)blockIdx.x < nlb) {  // the long rows, in the first warp's bitmap
    const int nl = *nlong;
    if ((int)blockIdx.x >= nl) return;
    for (int w = tid; w < nw; w += VT_WARPS * 32) vt_bitmap[w] = 0u;
    for (int i = blockIdx.x; i < nl; i += nlb) {
      const int q = longs[i], b = rowptr[q], cr = comp[q];
      const long long cell0 = (long long)(cr / V) * nseg;
      __syncthreads();
      set_bits(vt_bitmap, b, rowptr[q + 1] - b, tid, VT_WARPS * 32);
      __syncthreads();
      int n = 0;
      for (int w0 = 0; w0 < nw; w0 += VT_WARPS * 32) {
        const int w = w0 + tid;
        unsigned word = 0;
        if (w < nw) {
          word = vt_bitmap[w];
          vt_bitmap[w] = 0u;
        }
        const int c = nonzero_bytes(word), incl = warp_incl(c);
        if (lane == 31) wsum[warp] = incl;
        __syncthreads();
        int at = n + incl - c;
#pragma unroll
        for (int u = 0; u < VT_WARPS; ++u) {
          if (u < warp) at += wsum[u];
          n += wsum[u];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const unsigned bits = (word >> (8 * k)) & 0xffu;
          if (bits) emit(b, cell0, 4 * w + k, bits, at++);
        }
        __syncthreads();
      }
      if (tid == 0) tlist[cr] = make_int2(b, n);
    }
    return;
  }
  bool clean = false;  // this warp's bitmap is zero
  for (int q = ((int)blockIdx.x - nlb) * VT_WARPS + warp; q < m; q += ((int)gridDim.x - nlb) * VT_WARPS) {
    const int b = rowptr[q], len = rowptr[q + 1] - b;
    if (len > VT_LONG) continue;
    {
      const int cr = comp[q];
      const long long cell0 = (long long)(cr / V) * nseg;
      int n = 0;
      if (len <= 32) {
        unsigned key = lane < len ? (unsigned)packed[ccol[b + lane]] : ~0u;
#pragma unroll
        for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
          for (int j = k >> 1; j > 0; j >>= 1) {
            const unsigned other = __shfl_xor_sync(0xffffffffu, key, j);
            const bool up = (lane & k) == 0, low = (lane & j) == 0;
            key = (low == up) ? min(key, other) : max(key, other);
          }
        const unsigned s = key >> 3;
        const bool valid = key != ~0u;
        unsigned bits = valid ? 1u << (M - 1 - (int)(key & 7u)) : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {  // OR over the lanes of the same segment from here on
          const unsigned t = __shfl_down_sync(0xffffffffu, bits, o), ts = __shfl_down_sync(0xffffffffu, s, o);
          if (lane + o < 32 && ts == s) bits |= t;
        }
        const unsigned ps = __shfl_up_sync(0xffffffffu, s, 1);
        const unsigned heads = __ballot_sync(0xffffffffu, valid && (lane == 0 || ps != s));
        if ((heads >> lane) & 1u) emit(b, cell0, (int)s, bits, __popc(heads & ((1u << lane) - 1u)));
        n = __popc(heads);
      } else {
        if (!clean)
          for (int w = lane; w < nw; w += 32) bm[w] = 0u;
        clean = true;
        __syncwarp();
        unsigned touched = __reduce_or_sync(0xffffffffu, set_bits(bm, b, len, lane, 32));
        __syncwarp();
        for (; touched; touched &= touched - 1) {
          const int w0 = (__ffs(touched) - 1) * part, w1 = min(w0 + part, nw);
          for (int w = w0 + lane; w - lane < w1; w += 32) {
            unsigned word = 0;
            if (w < w1) {
              word = bm[w];
              bm[w] = 0u;
            }
            if (!__any_sync(0xffffffffu, word != 0u)) continue;
            const int c = nonzero_bytes(word), incl = warp_incl(c);
            int at = n + incl - c;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const unsigned bits = (word >> (8 * k)) & 0xffu;
              if (bits) emit(b, cell0, 4 * w + k, bits, at++);
            }
            n += __shfl_sync(0xffffffffu, incl, 31);
          }
        }
        __syncwarp();
      }
      if (lane == 0) tlist[cr] = make_int2(b, n);
    }
  }
}

// The stable order of the rows by their token lists, in the shared memory of
// one thread-block cluster: position p lives in block p / cap (cap a power of
// two).  A row is one 64-bit word, its sort key above its id (16 bits).
// First all rows are sorted by their first two tokens; then each level sorts
// the rows of a group (rows equal so far) by their next token and splits the
// groups; a row alone in its group, or at the end of its list, keeps its
// place.  Sorting is a stable radix sort of VO_BITS-bit digits (two cluster
// barriers a digit: each warp ranks its 32-row chunks with __match_any, the
// blocks exchange their digit counts, and every row goes straight to its
// place in the other buffer, in whichever block), or, where the largest group
// has at most VO_COUNT rows (on R-MAT 16384 76 after two tokens, 9 after
// three), every row counts the rows of its group that come before it.
// Bound by latency and the scattered stores between the blocks: 16384 rows on
// 16 blocks take 47 us (5 digits of 4 us, a split 2.5 us, a counted level 6
// us), where the multi-kernel radix sort took 23 us a digit.
constexpr int VO_BITS = 9, VO_BINS = 1 << VO_BITS, VO_THREADS = 1024, VO_WARPS = 32, VO_ITEMS = 4, VO_MAX_CTAS = 16;
constexpr int VO_COUNT = 256, VO_ID = 16;
constexpr int VO_MAX_CAP = VO_THREADS * VO_ITEMS;
static_assert(VO_MAX_CAP * VO_MAX_CTAS == VO_MAX_ROWS && VO_MAX_ROWS <= 1 << VO_ID, "all rows fit the largest cluster");
struct alignas(16) OrderSmem {
  uint16_t whist[VO_WARPS][VO_BINS];       // a warp's digit counts, then the counts of the warps before it
  uint32_t tot[VO_BINS / 2];               // this block's digit counts, two to a word
  uint32_t ctot[VO_MAX_CTAS][VO_BINS / 2]; // every block's
  int base[VO_BINS];                       // where this block's rows of a digit go
  int wsum[VO_WARPS];
  int wbig[VO_WARPS];
  int cmax[VO_MAX_CTAS];                   // every block's last group start,
  int cbig[VO_MAX_CTAS];                   // largest group that can still be split (0: none)
};

__global__ void __launch_bounds__(VO_THREADS, 1)
    k_vs_order(const int2* __restrict__ tlist, const unsigned* __restrict__ gtok, int m, int nseg, int tokbits,
               int grpbits, int cap, int* order) {
  extern __shared__ __align__(16) unsigned char vo_raw[];
  OrderSmem& sm = *reinterpret_cast<OrderSmem*>(vo_raw);
  auto* const buf = reinterpret_cast<unsigned long long*>(vo_raw + sizeof(OrderSmem));  // [2][cap]
  cg::cluster_group cl = cg::this_cluster();
  const int nct = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int capb = 31 - __clz(cap);
  const int items = cap / VO_THREADS;  // 32-row chunks a warp
  auto slot_of = [&](int j) { return (w * items + j) * 32 + lane; };  // of this lane's item j
  auto live_of = [&](int j) { return rank * cap + slot_of(j) < m; };
  const unsigned endtok = (unsigned)nseg << 8, idmask = (1u << VO_ID) - 1u;
  int cur = 0;

  // stable radix sort of the current buffer by bits VO_ID .. VO_ID + bits - 1
  auto radix = [&](int bits) {
    for (int shift = VO_ID; shift < VO_ID + bits; shift += VO_BITS) {
      const unsigned long long* key = buf + cur * cap;
      uint32_t* wh = reinterpret_cast<uint32_t*>(&sm.whist[0][0]);
      for (int i = tid; i < VO_WARPS * VO_BINS / 8; i += VO_THREADS)
        reinterpret_cast<uint4*>(wh)[i] = make_uint4(0u, 0u, 0u, 0u);
      __syncthreads();
      unsigned long long v[VO_ITEMS];
      int dig[VO_ITEMS], at[VO_ITEMS];
#pragma unroll
      for (int j = 0; j < VO_ITEMS; ++j) {
        if (j >= items) break;
        const bool live = live_of(j);
        v[j] = live ? key[slot_of(j)] : 0ull;
        dig[j] = live ? (int)(v[j] >> shift) & (VO_BINS - 1) : VO_BINS + lane;
        const unsigned peers = __match_any_sync(0xffffffffu, dig[j]);
        at[j] = live ? sm.whist[w][dig[j]] + __popc(peers & ((1u << lane) - 1u)) : 0;
        __syncwarp();
        if (live && lane == __ffs(peers) - 1) sm.whist[w][dig[j]] += (uint16_t)__popc(peers);
        __syncwarp();
      }
      __syncthreads();
      if (tid < VO_BINS / 2) {  // counts of the warps before, two digits a thread (no carry: at most cap)
        uint32_t run = 0;
#pragma unroll 8
        for (int u = 0; u < VO_WARPS; ++u) {
          const uint32_t c = wh[u * (VO_BINS / 2) + tid];
          wh[u * (VO_BINS / 2) + tid] = run;
          run += c;
        }
        sm.tot[tid] = run;
      }
      __syncthreads();
      for (int i = tid; i < nct * (VO_BINS / 2); i += VO_THREADS)
        *cl.map_shared_rank(&sm.ctot[rank][i % (VO_BINS / 2)], i / (VO_BINS / 2)) = sm.tot[i % (VO_BINS / 2)];
      cl.sync();
      if (tid < VO_BINS / 2) {
        int lo = 0, hi = 0, blo = 0, bhi = 0;  // all blocks' counts, and of the blocks before this one
        for (int c = 0; c < nct; ++c) {
          const uint32_t x = sm.ctot[c][tid];
          if (c == rank) {
            blo = lo;
            bhi = hi;
          }
          lo += (int)(x & 0xffffu);
          hi += (int)(x >> 16);
        }
        int incl = lo + hi;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += t;
        }
        if (lane == 31) sm.wsum[w] = incl;
        sm.base[2 * tid] = incl - lo - hi + blo;
        sm.base[2 * tid + 1] = incl - hi + bhi;
      }
      __syncthreads();
      unsigned long long* const out = buf + (cur ^ 1) * cap;
#pragma unroll
      for (int j = 0; j < VO_ITEMS; ++j)
        if (j < items && live_of(j)) {
          int before = 0;
          for (int u = 0; u < dig[j] >> 6; ++u) before += sm.wsum[u];
          const int dst = sm.base[dig[j]] + before + sm.whist[w][dig[j]] + at[j];
          *cl.map_shared_rank(out + (dst & (cap - 1)), dst >> capb) = v[j];
        }
      cl.sync();
      cur ^= 1;
    }
  };

  int grp[VO_ITEMS];     // start of the group of each of this lane's positions
  unsigned settled = 0;  // bit j: position j keeps its row
  // Split the groups: a row starts one when its key differs from the one
  // before, and is settled when it is alone in it or its list has ended
  // (ended(key)).  Returns the size of the largest group left to split.
  auto split = [&](auto&& ended) -> int {
    const unsigned long long* key = buf + cur * cap;
    int last = -1;  // the last group start up to here, of this warp
    unsigned alone = 0, done = 0, tails = 0;
#pragma unroll
    for (int j = 0; j < VO_ITEMS; ++j) {
      if (j >= items) break;
      const int sl = slot_of(j), pos = rank * cap + sl;
      int start = -1;
      if (live_of(j)) {
        const unsigned long long me = key[sl] >> VO_ID;
        const bool head =
            pos == 0 || me != (sl > 0 ? key[sl - 1] : *cl.map_shared_rank(key + cap - 1, rank - 1)) >> VO_ID;
        const bool tail =
            pos == m - 1 || me != (sl + 1 < cap ? key[sl + 1] : *cl.map_shared_rank(key, rank + 1)) >> VO_ID;
        if (head) start = pos;
        if (tail) tails |= 1u << j;
        if (head && tail) alone |= 1u << j;
        if (ended(me)) done |= 1u << j;
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, start, o);
        if (lane >= o) start = max(start, t);
      }
      grp[j] = max(start, last);
      last = max(last, __shfl_sync(0xffffffffu, start, 31));
    }
    settled = alone | done;
    if (lane == 0) sm.wsum[w] = last;
    __syncthreads();
    int mine = sm.wsum[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, mine, o);
      if (lane >= o) mine = max(mine, t);
    }
    const int all = __shfl_sync(0xffffffffu, mine, 31);
    int before = __shfl_sync(0xffffffffu, mine, w > 0 ? w - 1 : 0);
    if (w == 0) before = -1;
    if (tid < nct) *cl.map_shared_rank(&sm.cmax[rank], tid) = all;
    cl.sync();
    for (int c = 0; c < rank; ++c) before = max(before, sm.cmax[c]);
    int big = 0;
#pragma unroll
    for (int j = 0; j < VO_ITEMS; ++j) {
      if (j >= items) break;
      grp[j] = max(grp[j], before);
      if (((tails & ~settled) >> j) & 1u) big = max(big, rank * cap + slot_of(j) - grp[j] + 1);
    }
    big = __reduce_max_sync(0xffffffffu, big);
    if (lane == 0) sm.wbig[w] = big;
    __syncthreads();
    if (tid < nct) {
      int b = 0;
      for (int u = 0; u < VO_WARPS; ++u) b = max(b, sm.wbig[u]);
      *cl.map_shared_rank(&sm.cbig[rank], tid) = b;
    }
    cl.sync();
    int b = 0;
    for (int c = 0; c < nct; ++c) b = max(b, sm.cbig[c]);
    return b;
  };

#pragma unroll
  for (int j = 0; j < VO_ITEMS; ++j)
    if (j < items && live_of(j)) {
      const int r = rank * cap + slot_of(j);
      const int2 t = tlist[r];
      const unsigned t0 = t.y > 0 ? gtok[t.x] : endtok, t1 = t.y > 1 ? gtok[t.x + 1] : t.y == 1 ? endtok : 0u;
      buf[slot_of(j)] = ((unsigned long long)t0 << tokbits | t1) << VO_ID | (unsigned)r;
    }
  cl.sync();  // every block has started before any remote access
  radix(2 * tokbits);
  const unsigned tmask = (1u << tokbits) - 1u;
  int big = split([&](unsigned long long k) { return ((unsigned)k & tmask) == endtok || ((unsigned)k & tmask) == 0u; });
  for (int k = 2; big > 1; ++k) {
    // keys: the group, the next token (0 for a settled row)
    unsigned long long* key = buf + cur * cap;
    unsigned tok[VO_ITEMS];
#pragma unroll
    for (int j = 0; j < VO_ITEMS; ++j)
      if (j < items && live_of(j)) {
        const unsigned r = (unsigned)key[slot_of(j)] & idmask;
        tok[j] = 0;
        if (!((settled >> j) & 1u)) {
          const int2 t = tlist[r];
          tok[j] = k < t.y ? gtok[t.x + k] : endtok;
        }
        key[slot_of(j)] = ((unsigned long long)(unsigned)grp[j] << tokbits | tok[j]) << VO_ID | r;
      }
    cl.sync();
    if (big > VO_COUNT) {
      radix(tokbits + grpbits);
    } else {
      unsigned long long* const out = buf + (cur ^ 1) * cap;
#pragma unroll
      for (int j = 0; j < VO_ITEMS; ++j)
        if (j < items && live_of(j)) {
          const int pos = rank * cap + slot_of(j);
          int dst = pos;
          if (!((settled >> j) & 1u)) {
            auto at = [&](int p) {
              return (p >> capb) == rank ? key[p & (cap - 1)] : *cl.map_shared_rank(key + (p & (cap - 1)), p >> capb);
            };
            dst = grp[j];
            for (int p = grp[j]; p < pos; ++p) dst += ((unsigned)(at(p) >> VO_ID) & tmask) <= tok[j] ? 1 : 0;
            for (int p = pos + 1; p < m; ++p) {
              const unsigned long long o = at(p) >> VO_ID;
              if ((int)(o >> tokbits) != grp[j]) break;
              dst += ((unsigned)o & tmask) < tok[j] ? 1 : 0;
            }
          }
          *cl.map_shared_rank(out + (dst & (cap - 1)), dst >> capb) = key[slot_of(j)];
        }
      cl.sync();
      cur ^= 1;
    }
    big = split([&](unsigned long long q) { return ((unsigned)q & tmask) == endtok || ((unsigned)q & tmask) == 0u; });
  }
#pragma unroll
  for (int j = 0; j < VO_ITEMS; ++j)
    if (j < items && live_of(j)) order[rank * cap + slot_of(j)] = (int)((unsigned)buf[cur * cap + slot_of(j)] & idmask);
}

struct VnmRows {  // the original matrix by rows, and the state of the rounds
  int m, M, V, nseg, tokbits;
  long long ncells;
  int *rowptr, *ccol, *packed;
  int2* tlist;
  unsigned *gtok, *ortab, *badtab;
  int *counts, *order;
  int* longs;                 // how many rows of more than VT_LONG entries, and the rows
  int round = 0;              // analyses so far
  cudaLaunchConfig_t cfg;     // launch shape of k_vs_order
  cudaLaunchAttribute attr[1];
  int cap = 0;
};
constexpr int VO_COUNTS = 64;

static size_t vnm_rows_bytes(int mp, int np, int nnz, long long ncells) {
  const int nodes = mp > np ? mp : np;
  return arena_bytes(mp + 1, 4) * 3 + arena_bytes(nnz + 1, 4) * 2 + arena_bytes(nodes, 4) + arena_bytes(mp, 8) +
         2 * arena_bytes((ncells + 3) / 4 + 1, 4) + arena_bytes(64, 4) + arena_bytes(mp, 4) + scan_scratch_bytes(mp + 1) +
         4096;
}

static vnm_status vnm_rows_build(vnm_ctx* ctx, int mp, int np, int nnz, const int* row, const int* col, int M, int V,
                                 VnmRows& W) {
  W.m = mp;
  W.M = M;
  W.V = V;
  W.nseg = np / M;
  W.ncells = (long long)((mp + V - 1) / V) * W.nseg;
  W.tokbits = bits_for(2ll * W.nseg) + 8;
  W.rowptr = arena_take<int>(ctx, mp + 1);
  int* fill = arena_take<int>(ctx, mp + 1);
  W.ccol = arena_take<int>(ctx, nnz + 1);
  W.gtok = arena_take<unsigned>(ctx, nnz + 1);
  W.packed = arena_take<int>(ctx, mp > np ? mp : np);
  W.tlist = arena_take<int2>(ctx, mp);
  W.ortab = arena_take<unsigned>(ctx, (W.ncells + 3) / 4 + 1);
  W.badtab = arena_take<unsigned>(ctx, (W.ncells + 3) / 4 + 1);
  W.counts = arena_take<int>(ctx, VO_COUNTS);
  W.order = arena_take<int>(ctx, mp);
  W.longs = arena_take<int>(ctx, mp + 1);
  if (!W.longs || !W.rowptr || !fill || !W.ccol || !W.gtok || !W.packed || !W.tlist || !W.ortab || !W.badtab || !W.counts ||
      !W.order)
    return VNM_ERR_NOMEM;
  VNM_CUDA_TRY(cudaMemsetAsync(W.rowptr, 0, sizeof(int) * (mp + 1), ctx->stream));
  VNM_CUDA_TRY(cudaMemsetAsync(fill, 0, sizeof(int) * (mp + 1), ctx->stream));
  VNM_CUDA_TRY(cudaMemsetAsync(W.ortab, 0, ((W.ncells + 3) / 4) * 4, ctx->stream));
  VNM_CUDA_TRY(cudaMemsetAsync(W.badtab, 0, ((W.ncells + 3) / 4) * 4, ctx->stream));
  VNM_CUDA_TRY(cudaFuncSetAttribute(k_vs_tokens, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    VT_WARPS * ((VO_MAX_SEG + 3) / 4) * 4));
  if (nnz) VNM_LAUNCH(ctx, k_vs_rowcount, vs_grid(ctx, nnz), VS_NT, 0, row, nnz, W.rowptr);
  VNM_TRY(exclusive_scan(ctx, W.rowptr, W.rowptr, mp + 1, nullptr));
  if (nnz) VNM_LAUNCH(ctx, k_vs_rowfill, vs_grid(ctx, nnz), VS_NT, 0, row, col, nnz, W.rowptr, fill, W.ccol);
  VNM_CUDA_TRY(cudaMemsetAsync(W.longs, 0, sizeof(int), ctx->stream));
  if (mp) VNM_LAUNCH(ctx, k_vs_long, vs_grid(ctx, mp), VS_NT, 0, W.rowptr, mp, W.longs + 1, W.longs);
  return VNM_OK;
}

// Tokens and V-block counts under the map `comp` (W.packed holds its places);
// the counts come back in h[0..1].
static vnm_status vnm_rows_analyse(vnm_ctx* ctx, VnmRows& W, const int* comp, int* h) {
  if (W.m > 0)
    VNM_LAUNCH(ctx, k_vs_tokens, 2 * ctx->num_sms + vs_grid(ctx, (long long)W.m * 32), VT_WARPS * 32,
               (size_t)VT_WARPS * ((W.nseg + 3) / 4) * 4, W.rowptr, W.ccol, comp, W.packed, W.longs + 1, W.longs,
               2 * ctx->num_sms, W.m, W.M, W.nseg, W.V,
               W.tlist, W.gtok, W.ortab, W.badtab);
  int* counts = W.counts + 2 * W.round++ % VO_COUNTS;  // a pair of its own for each of the next rounds
  if (counts == W.counts) VNM_CUDA_TRY(cudaMemsetAsync(W.counts, 0, VO_COUNTS * sizeof(int), ctx->stream));
  VNM_LAUNCH(ctx, k_vs_count<true>, vs_grid(ctx, (W.ncells + 3) / 4), VS_NT, 0, W.ortab, W.badtab, W.ncells, counts);
  VNM_CUDA_TRY(cudaMemcpyAsync(h, counts, 2 * sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  VNM_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  return VNM_OK;
}

static size_t vo_smem(int cap) { return sizeof(OrderSmem) + (size_t)2 * cap * sizeof(unsigned long long); }

// Launch shape of k_vs_order for m rows: a block for each 1024 rows (1, 2, 4,
// 8 or 16, then more rows a block), fewer blocks where the GPU cannot hold
// the cluster; false when the rows do not fit any it can hold.
static bool vnm_order_shape(vnm_ctx* ctx, int m, cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, int& cap) {
  int nct = 1;
  while (nct < VO_MAX_CTAS && nct * VO_THREADS < m) nct *= 2;
  // The kernel's ceilings belong to the function, which every host thread
  // shares: always the largest shape's, so that no call lowers another's
  // between its launches.
  if (cudaFuncSetAttribute(k_vs_order, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)vo_smem(VO_MAX_CAP)) !=
          cudaSuccess ||
      cudaFuncSetAttribute(k_vs_order, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  cfg = cudaLaunchConfig_t{};
  cfg.blockDim = dim3(VO_THREADS);
  cfg.stream = ctx->stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  for (; nct >= 1; nct /= 2) {
    cap = VO_THREADS;
    while (nct * cap < m) cap *= 2;
    if (cap > VO_MAX_CAP) break;
    cfg.gridDim = dim3(nct);
    cfg.dynamicSmemBytes = vo_smem(cap);
    attr[0].val.clusterDim.x = (unsigned)nct;
    int fit = 0;
    if (cudaOccupancyMaxActiveClusters(&fit, k_vs_order, &cfg) == cudaSuccess && fit >= 1) return true;
    (void)cudaGetLastError();
  }
  return false;
}

// W.order = the stable row order of reordering.py:219 for the analysed rows.
static vnm_status vnm_rows_order(vnm_ctx* ctx, VnmRows& W) {
  VNM_CUDA_TRY(cudaLaunchKernelEx(&W.cfg, k_vs_order, (const int2*)W.tlist, (const unsigned*)W.gtok, W.m, W.nseg,
                                  W.tokbits, bits_for(W.m - 1), W.cap, W.order));
  ctx->launches++;
  return VNM_OK;
}

// Whether a call runs on the original rows: all rows fit a cluster the GPU
// can hold, and every column's new place (the row map's) lies in a segment.
// VNM_VS_ROWS=0 in the environment takes every call to the general path.
static bool vnm_rows_fit(vnm_ctx* ctx, int mp, int np, int M, VnmRows& W) {
  if (const char* e = getenv("VNM_VS_ROWS"))
    if (atoi(e) == 0) return false;
  if (mp > VO_MAX_ROWS || mp > np || np / M > VO_MAX_SEG || cudaSetDevice(ctx->device) != cudaSuccess) return false;
  return vnm_order_shape(ctx, mp, W.cfg, W.attr, W.cap);
}

}  // namespace vnm

using namespace vnm;

extern "C" {

vnm_status vnm_vnm_eval(vnm_ctx* ctx, int m, int n, int nnz, const int* row, const int* col, int mem, int M, int V,
                        int* out2) {
  VNM_TRY(vnm_args(ctx, m, n, nnz, row, col, mem, M, V));
  if (!out2) return VNM_ERR_ARG;
  const int mp = (m + M - 1) / M * M, np = (n + M - 1) / M * M;
  const long long ncells = (long long)((mp + V - 1) / V) * (np / M);
  VnmRows R;
  const bool rows = vnm_rows_fit(ctx, mp, np, M, R);
  VNM_TRY(arena_reserve(ctx, (rows ? vnm_rows_bytes(mp, np, nnz, ncells) + arena_bytes(mp > np ? mp : np, 4)
                                   : vnm_bytes(mp, nnz, ncells)) +
                                 2 * arena_bytes(nnz, 4) + arena_bytes(1, 4)));
  VNM_TRY(pinned_reserve(ctx, 64));
  VNM_TRY(begin_call(ctx));
  const int *d_row, *d_col;
  VNM_TRY(stage_in(ctx, row, nnz, mem, &d_row));
  VNM_TRY(stage_in(ctx, col, nnz, mem, &d_col));
  int* err = arena_take<int>(ctx, 1);
  if (!err) return VNM_ERR_NOMEM;
  VNM_CUDA_TRY(cudaMemsetAsync(err, 0, sizeof(int), ctx->stream));
  if (nnz) VNM_LAUNCH(ctx, k_vs_check, vs_grid(ctx, nnz), VS_NT, 0, d_row, d_col, nnz, mp, np, err);
  VNM_CUDA_TRY(cudaMemcpyAsync(ctx->h_pinned, err, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  VNM_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  if (ctx->h_pinned[0]) return VNM_ERR_RANGE;
  if (rows) {
    VNM_TRY(vnm_rows_build(ctx, mp, np, nnz, d_row, d_col, M, V, R));
    const int nodes = mp > np ? mp : np;
    int* comp = arena_take<int>(ctx, nodes);
    if (!comp) return VNM_ERR_NOMEM;
    VNM_LAUNCH(ctx, k_vs_map, vs_grid(ctx, nodes), VS_NT, 0, nullptr, nullptr, nodes, M, comp, R.packed);
    VNM_TRY(vnm_rows_analyse(ctx, R, comp, ctx->h_pinned));
  } else {
    VnmWork W;
    VNM_TRY(vnm_setup(ctx, m, n, nnz, M, V, W));
    VNM_TRY(vnm_analyse(ctx, d_row, d_col, W, ctx->h_pinned));
  }
  out2[0] = ctx->h_pinned[0];
  out2[1] = ctx->h_pinned[1];
  return end_call(ctx);
}

// vnm_vnm_reorder on the original rows: prev (accepted) and cur (candidate)
// are node maps; the entries are relabelled once, at the end.
static vnm_status reorder_rows(vnm_ctx* ctx, VnmRows& W, int mp, int np, int nnz, int* row, int* col, int mem, int M,
                               int V, int maxiter, int* out5, int* newpos) {
  const long long ncells = (long long)((mp + V - 1) / V) * (np / M);
  VNM_TRY(arena_reserve(ctx, vnm_rows_bytes(mp, np, nnz, ncells) + 2 * arena_bytes(nnz + 1, 4) +
                                 2 * arena_bytes(mp > np ? mp : np, 4) + arena_bytes(1, 4)));
  VNM_TRY(pinned_reserve(ctx, 64));
  VNM_TRY(begin_call(ctx));
  int* h = ctx->h_pinned;
  const int nodes = mp > np ? mp : np;
  int *d_row = row, *d_col = col;
  if (mem == VNM_MEM_HOST && nnz) {
    d_row = arena_take<int>(ctx, nnz);
    d_col = arena_take<int>(ctx, nnz);
    if (!d_row || !d_col) return VNM_ERR_NOMEM;
    VNM_CUDA_TRY(cudaMemcpyAsync(d_row, row, sizeof(int) * nnz, cudaMemcpyHostToDevice, ctx->stream));
    VNM_CUDA_TRY(cudaMemcpyAsync(d_col, col, sizeof(int) * nnz, cudaMemcpyHostToDevice, ctx->stream));
  }
  int* prev = arena_take<int>(ctx, nodes);
  int* cur = arena_take<int>(ctx, nodes);
  int* err = arena_take<int>(ctx, 1);
  if (!prev || !cur || !err) return VNM_ERR_NOMEM;
  VNM_CUDA_TRY(cudaMemsetAsync(err, 0, sizeof(int), ctx->stream));
  // columns index new_id[] (m entries), as in reordering.py:175-176
  if (nnz) VNM_LAUNCH(ctx, k_vs_check, vs_grid(ctx, nnz), VS_NT, 0, d_row, d_col, nnz, mp, mp < np ? mp : np, err);
  VNM_CUDA_TRY(cudaMemcpyAsync(h, err, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  VNM_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  if (h[0]) return VNM_ERR_RANGE;
  VNM_TRY(vnm_rows_build(ctx, mp, np, nnz, d_row, d_col, M, V, W));
  VNM_LAUNCH(ctx, k_vs_map, vs_grid(ctx, mp), VS_NT, 0, nullptr, nullptr, mp, M, prev, W.packed);
  VNM_TRY(vnm_rows_analyse(ctx, W, prev, h));
  const int init_inv = h[0], init_strict = h[1];
  int inv = init_inv, prev_inv = init_inv, prev_strict = init_strict;
  int round = 1;
  const int MAXITER = init_inv > maxiter ? init_inv : maxiter;  // reordering.py:209-210
  bool early = false;
  while (inv > 0 && round <= MAXITER) {
    VNM_TRY(vnm_rows_order(ctx, W));  // new_id[i] = sorted_data[i][0]
    VNM_LAUNCH(ctx, k_vs_map, vs_grid(ctx, mp), VS_NT, 0, prev, W.order, mp, M, cur, W.packed);
    VNM_TRY(vnm_rows_analyse(ctx, W, cur, h));
    inv = h[0];
    if (inv > prev_inv) {  // reordering.py:242-246: keep the previous state
      early = true;
      break;
    }
    prev_inv = inv;
    prev_strict = h[1];
    std::swap(prev, cur);
    round += 1;
  }
  out5[0] = init_inv;
  out5[1] = init_strict;
  out5[2] = prev_inv;
  out5[3] = prev_strict;
  out5[4] = early ? round : round - 1;
  if (nnz) {
    VNM_LAUNCH(ctx, k_vs_apply, vs_grid(ctx, nnz), VS_NT, 0, d_row, d_col, nnz, prev);
    if (mem == VNM_MEM_HOST) {
      VNM_CUDA_TRY(cudaMemcpyAsync(row, d_row, sizeof(int) * nnz, cudaMemcpyDeviceToHost, ctx->stream));
      VNM_CUDA_TRY(cudaMemcpyAsync(col, d_col, sizeof(int) * nnz, cudaMemcpyDeviceToHost, ctx->stream));
    }
  }
  if (newpos) VNM_CUDA_TRY(cudaMemcpyAsync(newpos, prev, sizeof(int) * mp, cudaMemcpyDeviceToHost, ctx->stream));
  return end_call(ctx);
}

vnm_status vnm_vnm_reorder(vnm_ctx* ctx, int m, int n, int nnz, int* row, int* col, int mem, int M, int V,
                           int maxiter, int* out5, int* newpos) {
  VNM_TRY(vnm_args(ctx, m, n, nnz, row, col, mem, M, V));
  if (!out5) return VNM_ERR_ARG;
  const int mp = (m + M - 1) / M * M, np = (n + M - 1) / M * M;
  const long long ncells = (long long)((mp + V - 1) / V) * (np / M);
  VnmRows R;
  if (vnm_rows_fit(ctx, mp, np, M, R))
    return reorder_rows(ctx, R, mp, np, nnz, row, col, mem, M, V, maxiter, out5, newpos);
  VNM_TRY(arena_reserve(ctx, vnm_bytes(mp, nnz, ncells)));
  VNM_TRY(pinned_reserve(ctx, 64));
  VNM_TRY(begin_call(ctx));
  int* h = ctx->h_pinned;
  // state: prev (accepted) and cur (candidate) COO + composed row maps
  int* prev_r = arena_take<int>(ctx, nnz > 0 ? nnz : 1);
  int* prev_c = arena_take<int>(ctx, nnz > 0 ? nnz : 1);
  int* cur_r = arena_take<int>(ctx, nnz > 0 ? nnz : 1);
  int* cur_c = arena_take<int>(ctx, nnz > 0 ? nnz : 1);
  int* prev_comp = arena_take<int>(ctx, mp);
  int* cur_comp = arena_take<int>(ctx, mp);
  int* err = arena_take<int>(ctx, 1);
  if (!prev_r || !prev_c || !cur_r || !cur_c || !prev_comp || !cur_comp || !err) return VNM_ERR_NOMEM;
  if (nnz) {
    const cudaMemcpyKind kind = mem == VNM_MEM_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
    VNM_CUDA_TRY(cudaMemcpyAsync(prev_r, row, sizeof(int) * nnz, kind, ctx->stream));
    VNM_CUDA_TRY(cudaMemcpyAsync(prev_c, col, sizeof(int) * nnz, kind, ctx->stream));
  }
  VNM_CUDA_TRY(cudaMemsetAsync(err, 0, sizeof(int), ctx->stream));
  // columns index new_id[] (m entries), as in reordering.py:175-176
  if (nnz) VNM_LAUNCH(ctx, k_vs_check, vs_grid(ctx, nnz), VS_NT, 0, prev_r, prev_c, nnz, mp, mp < np ? mp : np, err);
  VNM_CUDA_TRY(cudaMemcpyAsync(h, err, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  VNM_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  if (h[0]) return VNM_ERR_RANGE;
  VNM_LAUNCH(ctx, k_vs_iota, vs_grid(ctx, mp), VS_NT, 0, prev_comp, mp);
  VnmWork W;
  VNM_TRY(vnm_setup(ctx, m, n, nnz, M, V, W));
  VNM_TRY(vnm_analyse(ctx, prev_r, prev_c, W, h));
  const int init_inv = h[0], init_strict = h[1];
  int inv = init_inv, prev_inv = init_inv, prev_strict = init_strict;
  int round = 1;
  const int MAXITER = init_inv > maxiter ? init_inv : maxiter;  // reordering.py:209-210
  bool early = false;
  while (inv > 0 && round <= MAXITER) {
    // W holds the analysis of prev: sort its rows
    VNM_TRY(vnm_row_order(ctx, W, h));
    const int* new_id = W.order;  // new_id[i] = sorted_data[i][0]
    if (nnz) {
      VNM_CUDA_TRY(cudaMemcpyAsync(cur_r, prev_r, sizeof(int) * nnz, cudaMemcpyDeviceToDevice, ctx->stream));
      VNM_CUDA_TRY(cudaMemcpyAsync(cur_c, prev_c, sizeof(int) * nnz, cudaMemcpyDeviceToDevice, ctx->stream));
      VNM_LAUNCH(ctx, k_vs_apply, vs_grid(ctx, nnz), VS_NT, 0, cur_r, cur_c, nnz, new_id);
    }
    VNM_CUDA_TRY(cudaMemcpyAsync(cur_comp, prev_comp, sizeof(int) * mp, cudaMemcpyDeviceToDevice, ctx->stream));
    VNM_LAUNCH(ctx, k_vs_compose, vs_grid(ctx, mp), VS_NT, 0, cur_comp, mp, new_id);
    VNM_TRY(vnm_analyse(ctx, cur_r, cur_c, W, h));
    inv = h[0];
    const int istrict = h[1];
    if (inv > prev_inv) {  // reordering.py:242-246: keep the previous state
      early = true;
      break;
    }
    prev_inv = inv;
    prev_strict = istrict;
    std::swap(prev_r, cur_r);
    std::swap(prev_c, cur_c);
    std::swap(prev_comp, cur_comp);
    round += 1;
  }
  out5[0] = init_inv;
  out5[1] = init_strict;
  out5[2] = prev_inv;
  out5[3] = prev_strict;
  out5[4] = early ? round : round - 1;
  if (nnz) {
    const cudaMemcpyKind kind = mem == VNM_MEM_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice;
    VNM_CUDA_TRY(cudaMemcpyAsync(row, prev_r, sizeof(int) * nnz, kind, ctx->stream));
    VNM_CUDA_TRY(cudaMemcpyAsync(col, prev_c, sizeof(int) * nnz, kind, ctx->stream));
  }
  if (newpos) VNM_CUDA_TRY(cudaMemcpyAsync(newpos, prev_comp, sizeof(int) * mp, cudaMemcpyDeviceToHost, ctx->stream));
  return end_call(ctx);
}

}  // extern "C"
