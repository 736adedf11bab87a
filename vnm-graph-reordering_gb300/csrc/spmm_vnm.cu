// V:N:M SpMM: C = A * B with A sparse (the reordered matrix) and B dense,
// BF16 or FP16 operands, FP32 accumulation.  Dense V:N:M blocks run on the
// tcgen05 tensor cores; the blocks too sparse to pay for a tensor-core tile
// run on the CUDA cores.
//
// Replaces the reference's BSR WMMA kernel (kernel/spmm.cu:44-161), which
// runs one warp per 16x16 output tile with wmma m16n16k16 over 16x16 BSR
// blocks.  Here A is first compressed into its V:N:M layout and the dense
// products run as tcgen05.mma with the accumulator in tensor memory.
//
// Layout (the compressor below builds it on the device):
//   - rows are cut into tiles of 128 (the MMA's M); V must divide 128, so a
//     tile holds 128 / V block rows of V rows each.
//   - every non-empty (block row, segment) block -- V rows x M columns --
//     with at least `dense_min` nonzeros is cut into slices: 4 of its
//     columns, and per row at most 2 nonzeros among them (2:4 inside the
//     slice).  A block that satisfies V:N:M (at most 4 nonzero columns, at
//     most 2 nonzeros per row) is one slice; a block that does not spills
//     into more slices, so no nonzero is dropped and the product is exact up
//     to the operand rounding.
//   - 4 slices make one K-step of 16: the A operand of a K-step (128 rows x
//     16) is stored ready for the MMA (K-major, core matrices of 8 rows x 16
//     bytes), and the 16 B rows it multiplies are listed by index (-1 for a
//     column that only pads a slice: its B row is zero-filled, not read).
//   - values are stored divided by their block row's scale (max |a| of the
//     V rows), and the epilogue multiplies each output row back by it.
//   - the nonzeros of sparser blocks form the residual: a row-major CSR with
//     FP32 values, cut into tasks of at most 256 nonzeros of one row (a row
//     with more is split into chunks whose partial rows are added in a fixed
//     order afterwards, so the sums do not depend on timing).  No cap on the
//     chunks of a row: on a power-law graph (Chung-Lu 262144, max degree
//     72098, n=256) a cap of 32 left one warp walking 2254 entries while the
//     other SMs idled: 0.60 ms a product on GB300, 0.39 ms without the cap.
// On graph sparsity most blocks hold one or two nonzeros; a 128 x 16
// tensor-core tile for them would be >99 % padding, while a CUDA-core
// gather reads one B row per nonzero.  `dense_min` (VNM_SPMM_DENSE_MIN in the
// environment, else the default below) sets the split.
//
// Kernels of one product, in stream order:
//   k_spmm_res  CUDA cores: every residual task (and every row of a tile with
//               no tensor-core work) gathers its B rows with 16-byte loads and
//               writes its C row (or a partial row);
//   k_spmm_fin  adds the partial rows of the split rows, in chunk order;
//   k_spmm_vnm  tensor cores, one CTA per (work item, column block of C), a
//               work item being a tile's K-steps or a part of them.  Eight
//               producer warps stream stages of several K-steps: the A tiles
//               by one bulk copy, their B rows with 16-byte cp.async loads
//               into the 128-byte swizzled layout, the row ids loaded
//               several stages ahead; a ninth warp issues the MMAs.  The
//               producers then read the FP32 accumulator out of tensor
//               memory, scale it and store it, or add it to what the residual
//               wrote, or leave a part's sums for
//   k_spmm_tfin which adds the parts of the split tiles, in K order.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "sm100_ptx.cuh"

struct vnm_spmm_matrix {
  int device = 0;
  int R = 0, M = 0, V = 0, dtype = 1;  // dtype: 1 bf16, 0 f16
  int ntiles = 0, nsteps = 0;
  long long nnz = 0, groups = 0, slices = 0, slices_padded = 0, valid_blocks = 0;
  // tensor-core part
  int ntt = 0;                 // tiles with at least one K-step
  int npart = 0, ntsplit = 0, ntslots = 0;
  int4* part_list = nullptr;   // [npart] {2 tile + (1: the residual kernel wrote its rows first), begin, end, slot or -1}
  int4* tsplit = nullptr;      // [ntsplit] tiles cut into several parts: {2 tile + .., first slot, parts, 0}
  int* cols = nullptr;         // [nsteps * 16], -1 = padding column
  unsigned char* a = nullptr;  // [nsteps * 4096]
  float* rscale = nullptr;     // [ntiles * 128]
  // CUDA-core part
  int dense_min = 0;           // blocks with fewer nonzeros went to the residual
  long long nres = 0;          // residual nonzeros
  int ntask = 0, nmulti = 0, nslots = 0;
  int2* rcv = nullptr;         // [nres], row-major: {column, value bits}
  int4* task = nullptr;        // [ntask] {row, begin, end, partial slot or -1}
  int4* multi = nullptr;       // [nmulti] {row, first slot, chunks, 0}
  void* base = nullptr;        // one allocation for all of the above
  size_t bytes = 0;            // its size
  vnm_spmm_spare* spare = nullptr;  // the compressing context's spare storage
  // state of the asynchronous entry point
  float* part = nullptr;       // partial rows and tiles, for the largest n seen
  size_t part_floats = 0;
  bool part_own = false;       // an allocation of its own (the first PART_COLS columns' worth lies in `base`)
  int* err = nullptr;          // sticky failure flag of the tensor-core kernel
  bool pending = false;        // products were enqueued on a caller's stream, which nothing here waits for
};

namespace vnm {

constexpr int SP_TM = 128;        // rows per tile (MMA M)
constexpr int SP_KSTEP_BYTES = 4096;
constexpr int SP_THREADS = 288;
constexpr uint32_t SP_WAIT_LIMIT = 1u << 22;  // polls (each may suspend) before a wait gives up
constexpr uint32_t SP_SPIN_LIMIT = 1u << 26;  // polls of a pipeline wait, which spins
constexpr int RES_CHUNK = 256;    // residual nonzeros per task, at most
constexpr int RES_THREADS = 256;
constexpr int RES_U = 8;          // entries in flight per lane group (8 measured ahead of 4)
constexpr int RES_BLOCKS_PER_SM = 4;  // resident blocks of k_spmm_res an SM (64 registers a thread)
// A block runs on the tensor cores when it holds at least V nonzeros (one
// a row on average), else on the CUDA cores.  Measured on GB300 with the
// R-MAT 16384 (V=64, n=128) and Chung-Lu 262144 (V=128, n=256) operands,
// thresholds 2..64 against all-residual: every tensor-core share was slower
// (C2 0.037 ms all-residual vs 0.046-0.30 ms; C5 0.50 ms vs 0.67-4.9 ms):
// at one or two nonzeros per block a tile is >99 % padding and its fixed
// costs dominate.  A V:N:M operand whose blocks are full (2V nonzeros) goes
// to the tensor cores.  VNM_SPMM_DENSE_MIN overrides the threshold (0 =
// every block on the tensor cores).

static inline int sp_grid(const vnm_ctx* ctx, long long n, int nt = 256) {
  long long g = (n + nt - 1) / nt, cap = (long long)ctx->num_sms * 16;
  if (g > cap) g = cap;
  return g < 1 ? 1 : (int)g;
}

static inline int sp_bits(long long v) {
  int b = 1;
  while ((1ll << b) <= v) ++b;
  return b;
}

// ---------------------------------------------------------------------------
// Compressor
// ---------------------------------------------------------------------------
// An entry's sort key: its V x M block (block row, segment) in the high
// bits, then the row inside the block (bv = log2 V bits; V is a power of
// two) and the column inside the segment (bm = ceil(log2 M) bits), so that
// every field comes out with a shift and a mask.  Sorted, the keys order the
// entries by block, row, column.
__host__ __device__ inline int key_bits_m(int M) { return M <= 2 ? 1 : M <= 4 ? 2 : 3; }

// Keys, max |a| of each block row of V rows (the values' bits: non-negative
// floats order like them; one atomic for a warp of one block row, and none
// where the maximum so far is as large), and *unsorted = 1 where a row id
// decreases.
__global__ void k_cmp_keys(const int* row, const int* col, const float* val, int nnz, int M, int V, int nseg, int bm,
                           int bv, unsigned long long* keys, unsigned* bmax, int* unsorted) {
  bool down = false;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nnz; i += gridDim.x * blockDim.x) {
    const int r = row[i], c = col[i];
    const unsigned long long blk = (unsigned long long)(r >> bv) * nseg + (unsigned)(c / M);
    keys[i] = (((blk << bv) | (unsigned)(r & (V - 1))) << bm) | (unsigned)(c % M);
    down |= i > 0 && row[i - 1] > r;
    unsigned m = __float_as_uint(fabsf(val[i]));
    const unsigned am = __activemask();
    int same;
    __match_all_sync(am, r >> bv, &same);
    if (same) m = __reduce_max_sync(am, m);
    if ((!same || (int)(threadIdx.x & 31) == __ffs(am) - 1) && m > *(volatile unsigned*)&bmax[r >> bv])
      atomicMax(&bmax[r >> bv], m);
  }
  if (__syncthreads_or(down) && threadIdx.x == 0) atomicOr(unsorted, 1);
}

__device__ __forceinline__ unsigned low2(unsigned m) {  // the lowest two set bits of m
  const unsigned a = m & (0u - m);
  const unsigned rest = m & ~a;
  return a | (rest & (0u - rest));
}

// Counters of a compression.
constexpr int TASK_CLASSES = 7;  // of residual tasks, by length (task_class)
enum { CC_GROUPS, CC_VALID, CC_SLICES, CC_TILES, CC_RES, CC_MULTI_ROWS, CC_PADDED, CC_PARTS, CC_SPLIT, CC_SLOTS,
       CC_DENSE, CC_UNSORTED, CC_CLASS, CC_CURSOR = CC_CLASS + TASK_CLASSES, CC_MULTI_CURSOR = CC_CURSOR + TASK_CLASSES,
       CC_N };

// The blocks, each walked by the thread of its first entry (neighbouring
// threads walk neighbouring keys, so the walk lives in L1).  A block of fewer
// than dense_min nonzeros is residual: its entries are flagged (by original
// position) and counted per row, its tile marked.  A denser one goes to the
// list of dense blocks, which warps take over.  228 K entries in 200 K
// blocks: 22 us, where scanning block heads into a start table and one
// thread a block, dense ones included, took 115.
__global__ void __launch_bounds__(256)
    k_cmp_groups(const unsigned long long* __restrict__ skeys, const int* __restrict__ spos, int nnz, int V, int nseg,
                 int bm, int dense_min, int* dlist, int* resflag, int* rowlen, int* tile_res, int* counters) {
  const int sh = bm + __ffs(V) - 1;
  const unsigned omask = (1u << bm) - 1u;
  int groups = 0, valid = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nnz; i += gridDim.x * blockDim.x) {
    unsigned long long prev = skeys[i];
    const unsigned long long blk = prev >> sh;
    if (i > 0 && (skeys[i - 1] >> sh) == blk) continue;
    ++groups;
    // the walk: columns seen, and whether a row has more than 2 of them
    unsigned cols = 1u << ((unsigned)prev & omask);
    int n = 1, inrow = 1;
    bool bad = false;
    for (; n < dense_min && i + n < nnz; ++n) {
      const unsigned long long k = skeys[i + n];
      if ((k >> sh) != blk) break;
      cols |= 1u << ((unsigned)k & omask);
      if ((k >> bm) != (prev >> bm)) inrow = 1;
      else if (k != prev && ++inrow > 2) bad = true;
      prev = k;
    }
    if (n >= dense_min) {
      const unsigned am = __activemask();  // one atomic for the lanes that are here together
      const int lane = threadIdx.x & 31, lead = __ffs(am) - 1;
      int at = 0;
      if (lane == lead) at = atomicAdd(&counters[CC_DENSE], __popc(am));
      dlist[__shfl_sync(am, at, lead) + __popc(am & ((1u << lane) - 1u))] = i;
      continue;
    }
    valid += !bad && __popc(cols) <= 4;
    const int brow = (blk >> 32) == 0 ? (int)((unsigned)blk / (unsigned)nseg) : (int)(blk / (unsigned)nseg);
    for (int j = i; j < i + n; ++j) {
      resflag[spos[j]] = 1;
      atomicAdd(&rowlen[brow * V + ((int)(skeys[j] >> bm) & (V - 1))], 1);
    }
    tile_res[(brow * V) / SP_TM] = 1;
  }
  __shared__ int sum[2];
  if (threadIdx.x < 2) sum[threadIdx.x] = 0;
  __syncthreads();
  groups = __reduce_add_sync(0xffffffffu, groups);
  valid = __reduce_add_sync(0xffffffffu, valid);
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&sum[0], groups);
    atomicAdd(&sum[1], valid);
  }
  __syncthreads();
  if (threadIdx.x < 2 && sum[threadIdx.x]) atomicAdd(&counters[threadIdx.x == 0 ? CC_GROUPS : CC_VALID], sum[threadIdx.x]);
}

// A dense block on one warp: lane l holds the masks of its rows 4 l .. 4 l + 3,
// a byte each (bit o = column offset o), and smem the first entry of each row.
struct DenseBlock {
  unsigned mask;  // as above
  int n;          // entries
  int brow, seg;
};
constexpr int DB_WARPS = 8;
struct DenseSmem {
  unsigned mask[32];
  int first[SP_TM];
};

__device__ __forceinline__ DenseBlock load_dense(const unsigned long long* skeys, int b0, int nnz, int V, int nseg,
                                                 int bm, DenseSmem& sm) {
  const int lane = threadIdx.x & 31, sh = bm + __ffs(V) - 1;
  const unsigned long long blk = skeys[b0] >> sh;
  DenseBlock d;
  d.brow = (int)(blk / nseg);
  d.seg = (int)(blk % nseg);
  d.n = 0;
  sm.mask[lane] = 0u;
  __syncwarp();
  unsigned long long before = ~0ull;  // the key before this lane's
  for (int i0 = b0;; i0 += 32) {
    const int i = i0 + lane;
    const unsigned long long k = i < nnz ? skeys[i] : ~0ull;
    const bool in = i < nnz && (k >> sh) == blk;
    const unsigned long long up = __shfl_up_sync(0xffffffffu, k, 1);
    const unsigned long long prev = lane > 0 ? up : before;
    if (in) {
      const int r = (int)(k >> bm) & (V - 1);
      atomicOr(&sm.mask[r >> 2], (1u << ((unsigned)k & ((1u << bm) - 1u))) << (8 * (r & 3)));
      if (i == b0 || (prev >> bm) != (k >> bm)) sm.first[r] = i;
    }
    before = __shfl_sync(0xffffffffu, k, 31);
    const unsigned m = __ballot_sync(0xffffffffu, in);
    d.n += __popc(m);
    if (m != 0xffffffffu) break;
  }
  __syncwarp();
  d.mask = sm.mask[lane];
  __syncwarp();
  return d;
}

// The slices of one block, formed greedily: take the (up to) 4 columns with
// the most remaining nonzeros (ties to the lower offset), give each row at
// most 2 of its remaining nonzeros among them (lowest offsets first), repeat
// until the block is empty.  `emit(chosen, take)` is called once a slice with
// the chosen offsets and what each of the lane's rows takes.
template <class Emit>
__device__ __forceinline__ int dense_slices(unsigned mask, Emit&& emit) {
  int ns = 0;
  for (int guard = 0; guard < 64; ++guard) {
    int cnt[8], any = 0;
#pragma unroll
    for (int o = 0; o < 4; ++o) {  // two counts a word: at most 128 rows
      const int c = __reduce_add_sync(0xffffffffu, __popc(mask & (0x01010101u << o)) |
                                                       __popc(mask & (0x10101010u << o)) << 16);
      cnt[o] = c & 0xffff;
      cnt[o + 4] = c >> 16;
      any |= c;
    }
    if (!any) break;
    unsigned chosen = 0;
#pragma unroll
    for (int pick = 0; pick < 4; ++pick) {
      int best = 0, bo = -1;
#pragma unroll
      for (int o = 0; o < 8; ++o)
        if (!((chosen >> o) & 1u) && cnt[o] > best) {
          best = cnt[o];
          bo = o;
        }
      if (bo >= 0) chosen |= 1u << bo;
    }
    unsigned take = 0;
#pragma unroll
    for (int b = 0; b < 4; ++b) take |= low2((mask >> (8 * b)) & chosen) << (8 * b);
    emit(chosen, take);
    mask &= ~take;
    ++ns;
  }
  return ns;
}

// Slices of every dense block (at its first entry's place), per tile, and the
// blocks that satisfy V:N:M.
__global__ void __launch_bounds__(DB_WARPS * 32)
    k_cmp_dense(const unsigned long long* __restrict__ skeys, const int* __restrict__ dlist, int nnz, int V, int nseg,
                int bm, int* gsl, int* tile_raw, int* counters) {
  __shared__ DenseSmem sm[DB_WARPS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nd = counters[CC_DENSE];
  int nvalid = 0;
  for (int g = blockIdx.x * DB_WARPS + warp; g < nd; g += gridDim.x * DB_WARPS) {
    const int b0 = dlist[g];
    const DenseBlock d = load_dense(skeys, b0, nnz, V, nseg, bm, sm[warp]);
    const unsigned ors = __reduce_or_sync(0xffffffffu, d.mask);
    bool bad = false;
#pragma unroll
    for (int b = 0; b < 4; ++b) bad |= __popc((d.mask >> (8 * b)) & 0xffu) > 2;
    const bool valid = !__any_sync(0xffffffffu, bad) &&
                       __popc((ors | ors >> 8 | ors >> 16 | ors >> 24) & 0xffu) <= 4;
    const int ns = dense_slices(d.mask, [](unsigned, unsigned) {});
    if (lane == 0) {
      gsl[b0] = ns;
      atomicAdd(&tile_raw[(d.brow * V) / SP_TM], ns);
      nvalid += valid;
    }
  }
  if (nvalid) atomicAdd(&counters[CC_VALID], nvalid);
}

// Exclusive block-wide sums of N values a thread (1024 threads), each over
// all threads; `tot` gets the totals.
template <int N>
__device__ __forceinline__ void block_scan(int (&v)[N], int (&tot)[N]) {
  __shared__ int wsum[N][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int incl[N];
#pragma unroll
  for (int k = 0; k < N; ++k) {
    incl[k] = v[k];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, incl[k], o);
      if (lane >= o) incl[k] += x;
    }
    if (lane == 31) wsum[k][w] = incl[k];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < N; ++k) {
    int x = wsum[k][lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    tot[k] = __shfl_sync(0xffffffffu, x, 31);
    const int before = __shfl_sync(0xffffffffu, x, w > 0 ? w - 1 : 0);
    v[k] = incl[k] - v[k] + (w > 0 ? before : 0);
  }
  __syncthreads();  // wsum is free again
}

// How the tensor-core work of `steps` K-steps of a tile is cut: parts of
// about `per` K-steps, so that a few heavy tiles fill the chip.
__host__ __device__ __forceinline__ int tile_parts(int steps, int per) {
  const int k = (steps + per / 2) / per;
  return k < 1 ? 1 : k;
}
// K-steps a part: an even share of an SM, but no less than PART_MIN.  A part
// costs a CTA's set-up and the write and read of its partial tile, about as
// much as 30 K-steps: without parts, 32 tiles of 256 K-steps (4096 rows,
// V:2:8, V = 64) left 120 SMs idle (55 us a product at n = 128), and a hub
// tile of a Chung-Lu graph held the chip for 170 us.
constexpr int PART_MIN = 32;
constexpr int PART_COLS = 256;                       // columns whose partial sums an operand has room for from the start,
constexpr size_t PART_BYTES_MAX = size_t(256) << 20;  // unless they would take more than this

// One block plans the tiles: a tile's first slice (padded, and as counted),
// its first work item and their number, its place among the split tiles and
// its first partial slot; and their totals.
__global__ void __launch_bounds__(1024)
    k_tile_plan(const int* tile_raw, int ntiles, int num_sms, int* tile_base, int* tile_rawbase, int4* tile_plan,
                int* counters) {
  int run_pad = 0, run_raw = 0, run_has = 0;
  for (int t0 = 0; t0 <= ntiles; t0 += 1024) {
    const int t = t0 + threadIdx.x;
    const int raw = t < ntiles ? tile_raw[t] : 0;
    int v[3] = {(raw + 3) & ~3, raw, raw > 0 ? 1 : 0}, tot[3];
    block_scan<3>(v, tot);
    if (t <= ntiles) {
      tile_base[t] = run_pad + v[0];
      tile_rawbase[t] = run_raw + v[1];
    }
    run_pad += tot[0];
    run_raw += tot[1];
    run_has += tot[2];
  }
  const int total = run_pad / 4;  // K-steps
  const int share = (total + num_sms - 1) / num_sms, per = share > PART_MIN ? share : PART_MIN;
  int np = 0, ns = 0, nslot = 0;
  for (int t0 = 0; t0 < ntiles; t0 += 1024) {
    const int t = t0 + threadIdx.x;
    const int steps = t < ntiles ? (tile_raw[t] + 3) / 4 : 0;
    const int k = steps > 0 ? tile_parts(steps, per) : 0;
    int v[3] = {k, k > 1 ? 1 : 0, k > 1 ? k : 0}, tot[3];
    block_scan<3>(v, tot);
    if (t < ntiles) tile_plan[t] = make_int4(np + v[0], k, ns + v[1], nslot + v[2]);
    np += tot[0];
    ns += tot[1];
    nslot += tot[2];
  }
  if (threadIdx.x == 0) {
    counters[CC_SLICES] = run_raw;
    counters[CC_TILES] = run_has;
    counters[CC_PADDED] = run_pad;
    counters[CC_PARTS] = np;
    counters[CC_SPLIT] = ns;
    counters[CC_SLOTS] = nslot;
  }
}

// The residual entries in their original order, keyed by row for the
// stable sort that makes the CSR.
__global__ void k_res_compact(const int* resflag, const int* rpos, const int* row, int nnz, unsigned long long* rkey,
                              int* rsrc) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nnz; i += gridDim.x * blockDim.x)
    if (resflag[i]) {
      rkey[rpos[i]] = (unsigned long long)(unsigned)row[i];
      rsrc[rpos[i]] = i;
    }
}

__global__ void k_res_gather(const int* src, const int* col, const float* val, int nres, int2* rcv) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nres; i += gridDim.x * blockDim.x) {
    const int e = src[i];
    rcv[i] = make_int2(col[e], __float_as_int(val[e]));
  }
}

// Residual tasks of a row: none when its tile runs on the tensor cores and
// holds no residual entry (the tensor kernel then writes the rows), else one
// per chunk of at most RES_CHUNK entries (one task for an empty row, which
// writes zeros).
__device__ __forceinline__ int res_chunks(int len, bool needed) {
  if (!needed) return 0;
  return len <= RES_CHUNK ? 1 : (len + RES_CHUNK - 1) / RES_CHUNK;
}

// Class of a row's tasks, the longest first: the chunks of a split row, then
// whole rows by length.  The task list holds the classes in turn (the order
// inside one does not matter), so that the warps that walk it with one stride
// work on tasks of like length: with whole rows in row order the last warps of
// a Chung-Lu 262144 product ran 18 % longer than the average.
__device__ __forceinline__ int task_class(int len, int nch) {
  return nch > 1 ? 0 : len > 64 ? 1 : len > 32 ? 2 : len > 16 ? 3 : len > 8 ? 4 : len > 4 ? 5 : 6;
}

// The residual rows in tiles of RP_TILE rows: sums[t] = entries of tile t;
// tasks of each class, entries and split rows in the counters.
constexpr int RP_TILE = 1024;
__device__ __forceinline__ int2 res_of_row(int r, int R, const int* rowlen, const int* tile_raw, const int* tile_res) {
  if (r >= R) return make_int2(0, 0);
  const int t = r / SP_TM, len = rowlen[r];
  return make_int2(len, res_chunks(len, !(tile_raw[t] > 0 && tile_res[t] == 0)));
}

__global__ void __launch_bounds__(RP_TILE)
    k_res_plan(const int* rowlen, int R, const int* tile_raw, const int* tile_res, int* sums, int* counters) {
  __shared__ int cls[TASK_CLASSES + 2];
  if (threadIdx.x < TASK_CLASSES + 2) cls[threadIdx.x] = 0;
  __syncthreads();
  const int2 x = res_of_row(blockIdx.x * RP_TILE + threadIdx.x, R, rowlen, tile_raw, tile_res);
  if (x.y) atomicAdd(&cls[task_class(x.x, x.y)], x.y);
  if (x.y > 1) atomicAdd(&cls[TASK_CLASSES], 1);
  const int len = __reduce_add_sync(0xffffffffu, x.x);
  if ((threadIdx.x & 31) == 0 && len) atomicAdd(&cls[TASK_CLASSES + 1], len);
  __syncthreads();
  if (threadIdx.x < TASK_CLASSES + 2 && cls[threadIdx.x])
    atomicAdd(&counters[threadIdx.x < TASK_CLASSES ? CC_CLASS + threadIdx.x
                        : threadIdx.x == TASK_CLASSES ? CC_MULTI_ROWS : CC_RES], cls[threadIdx.x]);
  if (threadIdx.x == 0) sums[blockIdx.x] = cls[TASK_CLASSES + 1];
}

// The tasks; a split row's chunks are neighbours, and its partial slots are
// their places in the list.
__global__ void __launch_bounds__(RP_TILE)
    k_res_tasks(const int* rowlen, int R, const int* tile_raw, const int* tile_res, const int* sums, int* counters,
                int4* task, int4* multi) {
  __shared__ int cls[TASK_CLASSES + 1], at[TASK_CLASSES + 1];
  int before[1] = {0}, off[1], tot[1];
  for (int t = threadIdx.x; t < (int)blockIdx.x; t += RP_TILE) before[0] += sums[t];
  block_scan<1>(before, off);  // entries of the tiles before this one
  if (threadIdx.x <= TASK_CLASSES) cls[threadIdx.x] = 0;
  __syncthreads();
  const int r = blockIdx.x * RP_TILE + threadIdx.x;
  const int2 x = res_of_row(r, R, rowlen, tile_raw, tile_res);
  const int c = task_class(x.x, x.y);
  const int in = x.y ? atomicAdd(&cls[c], x.y) : 0, inm = x.y > 1 ? atomicAdd(&cls[TASK_CLASSES], 1) : 0;
  int v[1] = {x.x};
  block_scan<1>(v, tot);
  if (threadIdx.x <= TASK_CLASSES) {
    int start = 0;
    for (int k = 0; k < (int)threadIdx.x && threadIdx.x < TASK_CLASSES; ++k) start += counters[CC_CLASS + k];
    const int n = cls[threadIdx.x];
    at[threadIdx.x] =
        start + (n ? atomicAdd(&counters[threadIdx.x < TASK_CLASSES ? CC_CURSOR + threadIdx.x : CC_MULTI_CURSOR], n) : 0);
  }
  __syncthreads();
  if (!x.y) return;
  const int b = off[0] + v[0], e = b + x.x, base = at[c] + in;
  if (x.y == 1) {
    task[base] = make_int4(r, b, e, -1);
    return;
  }
  const int csz = (x.x + x.y - 1) / x.y;
  for (int j = 0; j < x.y; ++j) {
    const int cb = min(b + j * csz, e), ce = min(cb + csz, e);
    task[base + j] = make_int4(r, cb, ce, base + j);
  }
  multi[at[TASK_CLASSES] + inm] = make_int4(r, base, x.y, 0);
}

// The residual records of entries that are sorted by row already.
__global__ void k_res_sorted(const int* resflag, const int* rpos, const int* col, const float* val, int nnz, int2* rcv) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nnz; i += gridDim.x * blockDim.x)
    if (resflag[i]) rcv[rpos[i]] = make_int2(col[i], __float_as_int(val[i]));
}

// The work items of the tiles with K-steps, split tiles' parts in K order.
__global__ void k_tile_parts(const int* tile_raw, const int* tile_res, int ntiles, const int* tile_base,
                             const int4* tile_plan, int4* part, int4* tsplit) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < ntiles; t += gridDim.x * blockDim.x) {
    const int steps = (tile_raw[t] + 3) / 4, s0 = tile_base[t] / 4, x = 2 * t + (tile_res[t] > 0 ? 1 : 0);
    const int4 pl = tile_plan[t];
    for (int k = 0; k < pl.y; ++k)
      part[pl.x + k] = make_int4(x, s0 + (int)((long long)steps * k / pl.y), s0 + (int)((long long)steps * (k + 1) / pl.y),
                                 pl.y > 1 ? pl.w + k : -1);
    if (pl.y > 1) tsplit[pl.z] = make_int4(x, pl.w, pl.y, 0);
  }
}

template <class T>
__device__ __forceinline__ T to_t(float x);
template <>
__device__ __forceinline__ __nv_bfloat16 to_t<__nv_bfloat16>(float x) {
  return __float2bfloat16_rn(x);
}
template <>
__device__ __forceinline__ __half to_t<__half>(float x) {
  return __float2half_rn(x);
}

// Write every dense block's slices: B-row indices and A values in MMA layout,
// a row's 4 values of a slice (8 bytes) at once.  `gofs`: the slices of the
// blocks before, over all tiles.
template <class T>
__global__ void __launch_bounds__(DB_WARPS * 32)
    k_cmp_fill(const unsigned long long* __restrict__ skeys, const int* __restrict__ spos,
               const float* __restrict__ val, const int* __restrict__ dlist, int nd, int nnz, int M, int V, int nseg,
               int bm, const int* __restrict__ gofs, const int* __restrict__ tile_base,
               const int* __restrict__ tile_rawbase, const unsigned* __restrict__ bmax, int* cols, unsigned char* a) {
  __shared__ DenseSmem sm[DB_WARPS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int g = blockIdx.x * DB_WARPS + warp; g < nd; g += gridDim.x * DB_WARPS) {
    const int b0 = dlist[g];
    const DenseBlock d = load_dense(skeys, b0, nnz, V, nseg, bm, sm[warp]);
    const int t = (d.brow * V) / SP_TM;
    const float scale = bmax[d.brow] ? __uint_as_float(bmax[d.brow]) : 1.0f;
    const float inv = 1.0f / scale;
    int si = tile_base[t] + (gofs[b0] - tile_rawbase[t]);  // this block's first slice
    dense_slices(d.mask, [&](unsigned chosen, unsigned take) {
      const int ks = si >> 2, j = si & 3;
      if (lane < 4) {  // the lane-th chosen offset
        unsigned c = chosen;
        for (int q = 0; q < lane; ++q) c &= c - 1u;
        cols[ks * 16 + 4 * j + lane] = c ? d.seg * M + __ffs(c) - 1 : -1;
      }
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const unsigned tk = (take >> (8 * b)) & 0xffu, orig = (d.mask >> (8 * b)) & 0xffu;
        if (!tk) continue;
        const int rin = 4 * lane + b, rt = d.brow * V - t * SP_TM + rin;  // row inside the block, the tile
        alignas(8) T v[4];
        unsigned c = chosen;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const unsigned bit = c & (0u - c);
          c ^= bit;
          float x = 0.f;
          if (bit & tk) x = val[spos[sm[warp].first[rin] + __popc(orig & (bit - 1u))]] * inv;
          v[q] = to_t<T>(x);
        }
        const int off = (rt >> 3) * 256 + (j >> 1) * 128 + (rt & 7) * 16 + (j & 1) * 8;
        *reinterpret_cast<uint2*>(a + (size_t)ks * SP_KSTEP_BYTES + off) = *reinterpret_cast<const uint2*>(v);
      }
      ++si;
    });
    __syncwarp();  // `first` is read before the next block's writes
  }
}

__global__ void k_cmp_rscale(const unsigned* bmax, int ntiles, int R, int V, float* rscale) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ntiles * SP_TM; i += gridDim.x * blockDim.x) {
    const unsigned m = i < R ? bmax[i / V] : 0u;
    rscale[i] = m ? __uint_as_float(m) : 1.0f;
  }
}

// ---------------------------------------------------------------------------
// Residual kernels (CUDA cores)
// ---------------------------------------------------------------------------
// acc[0..3] (4 pairs of FP32 accumulators, packed two to a 64-bit register,
// element 0 in the low half) += w * the 8 16-bit values in b (element 0 in
// the low half of b.x), as four packed FP32 FMAs (fma.rn.f32x2: two
// round-to-nearest FP32 FMAs, the same results as eight scalar ones in half
// the instructions); ww is w in both halves.  The accumulators stay packed
// for a whole task.
template <bool BF16>
__device__ __forceinline__ void fma8(unsigned long long (&acc)[4], uint4 b, unsigned long long ww) {
  const uint32_t q[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint32_t lo, hi;
    if (BF16) {
      lo = q[i] << 16;
      hi = q[i] & 0xffff0000u;
    } else {
      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&q[i]));
      lo = __float_as_uint(f.x);
      hi = __float_as_uint(f.y);
    }
    unsigned long long xx;
    asm("mov.b64 %0, {%1, %2};" : "=l"(xx) : "r"(lo), "r"(hi));
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i]) : "l"(ww), "l"(xx));
  }
}

// A warp walks the task list with a stride of every warp of the grid (one
// wave of resident blocks); LW lanes cover the block's 8 * LW columns, 8
// consecutive ones a lane, and the G = 32 / LW groups of lanes take the
// task's records in turn, two at a time, their sums added at the end.  The
// records come 32 at a time, one a lane, through shared memory (a 16-byte
// read hands a group two of them; handing out columns and weights by shuffles
// cost two a record), the next 32, and the next task with its first 32, loaded
// ahead.  Every lane gathers its 16 bytes of RES_U rows before the first is
// used; a short rest of a task issues half as many.
// Bound by instructions issued (unpacking 16-bit values, packed FMAs, an
// address and a load a record and lane) and, next, the gathers from L2: 4.2 M
// records, n = 256 (Chung-Lu 262144): 234 us, 9.2 TB/s of gathered rows, 361
// with the records handed out by shuffles, padded batches of 8 and whole rows
// in row order (task_class).
template <bool BF16, int NU, bool FULL, int G>
__device__ __forceinline__ void res_step(unsigned long long (&acc)[4], const int4* rec, int grp, int left,
                                         const unsigned char* bcol, unsigned ldb) {
  uint4 b[NU];
  int w[NU];
#pragma unroll
  for (int u = 0; u < NU; u += 2) {
    const int4 r = rec[u / 2 * G + grp];  // records u * G + 2 grp and the one after it
    const int k = u * G + 2 * grp;
    const unsigned char *p0, *p1;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(p0) : "r"(r.x), "r"(ldb), "l"(bcol));
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(p1) : "r"(r.z), "r"(ldb), "l"(bcol));
    b[u] = FULL || k < left ? __ldg(reinterpret_cast<const uint4*>(p0)) : make_uint4(0, 0, 0, 0);
    b[u + 1] = FULL || k + 1 < left ? __ldg(reinterpret_cast<const uint4*>(p1)) : make_uint4(0, 0, 0, 0);
    w[u] = r.y;
    w[u + 1] = r.w;
  }
#pragma unroll
  for (int u = 0; u < NU; ++u) {
    unsigned long long ww;
    asm("mov.b64 %0, {%1, %1};" : "=l"(ww) : "r"(w[u]));
    fma8<BF16>(acc, b[u], ww);
  }
}

template <int LW, bool BF16>
__device__ __forceinline__ void res_tasks(const int4* __restrict__ task, int ntask, const int2* __restrict__ rcv,
                                          const unsigned char* __restrict__ B, unsigned ldb, float* __restrict__ C,
                                          int ldc, float* __restrict__ P, int ldp, int col0,
                                          int2 (*recs)[2][32]) {
  constexpr int G = 32 / LW;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, grp = lane / LW, lid = lane % LW;
  const int stride = gridDim.x * (RES_THREADS / 32);
  const int cb = col0 + lid * 8;  // this lane's first column
  const unsigned char* bcol = B + (size_t)cb * 2;
  int t = blockIdx.x * (RES_THREADS / 32) + warp, par = 0;
  if (t >= ntask) return;
  int4 tk = task[t];
  int2 rc = tk.y + lane < tk.z ? __ldg(rcv + tk.y + lane) : make_int2(0, 0);
  int4 tkn = t + stride < ntask ? task[t + stride] : make_int4(0, 0, 0, -1);
  for (; t < ntask; t += stride) {
    const int len = tk.z - tk.y;
    // the next task's first records, and the task after it
    const int2 rc1 = tkn.y + lane < tkn.z ? __ldg(rcv + tkn.y + lane) : make_int2(0, 0);
    const int4 tk2 = t + 2 * stride < ntask ? task[t + 2 * stride] : make_int4(0, 0, 0, -1);
    unsigned long long acc[4] = {0ull, 0ull, 0ull, 0ull};  // FP32 pairs
    for (int k0 = 0; k0 < len; k0 += 32) {
      recs[warp][par][lane] = rc;
      const int kn = k0 + 32 + lane;
      rc = kn < len ? __ldg(rcv + tk.y + kn) : make_int2(0, 0);
      __syncwarp();
      const int cnt = min(32, len - k0);
      const int4* rec = reinterpret_cast<const int4*>(recs[warp][par]);
#pragma unroll 1
      for (int s = 0; s < cnt; s += RES_U * G) {
        const int left = cnt - s;
        if (left >= RES_U * G) res_step<BF16, RES_U, true, G>(acc, rec + s / 2, grp, left, bcol, ldb);
        else if (left > RES_U * G / 2) res_step<BF16, RES_U, false, G>(acc, rec + s / 2, grp, left, bcol, ldb);
        else res_step<BF16, RES_U / 2, false, G>(acc, rec + s / 2, grp, left, bcol, ldb);
      }
      par ^= 1;  // (the other half is read before this one is written again)
    }
    float f[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      f[2 * i] = __uint_as_float((uint32_t)acc[i]);
      f[2 * i + 1] = __uint_as_float((uint32_t)(acc[i] >> 32));
    }
#pragma unroll
    for (int o = 16; o >= LW; o >>= 1)
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] += __shfl_xor_sync(0xffffffffu, f[i], o);
    float4* dst = reinterpret_cast<float4*>(tk.w < 0 ? C + (size_t)tk.x * ldc + cb : P + (size_t)tk.w * ldp + cb);
    if (G == 1 || grp == 0) dst[0] = make_float4(f[0], f[1], f[2], f[3]);
    if (G == 1 || grp == 1) dst[1] = make_float4(f[4], f[5], f[6], f[7]);
    tk = tkn;
    tkn = tk2;
    rc = rc1;
  }
}

// The column blocks of a product's C: 256 columns each, then one of 128 and one
// of 64 where they are left.  All in one launch: the blocks of the next
// width start where the ones before leave the SMs, and a small operand's
// widths run beside one another.  (A launch a width put their times end to
// end: 4096 rows, 64 K records, n = 192 / 320 / 448: 40 / 51 / 71 us, 25 / 34 / 35 now.)
static inline int col_blocks(int n) { return n / 256 + (n % 256) / 128 + (n % 128) / 64; }

template <bool BF16>
__global__ void __launch_bounds__(RES_THREADS, RES_BLOCKS_PER_SM)
    k_spmm_res(const int4* __restrict__ task, int ntask, const int2* __restrict__ rcv,
               const unsigned char* __restrict__ B, unsigned ldb, float* __restrict__ C, int ldc,
               float* __restrict__ P, int ldp) {
  __shared__ __align__(16) int2 recs[RES_THREADS / 32][2][32];
  const int col0 = blockIdx.y * 256, left = ldc - col0;  // (ldc: the columns of C)
  if (left >= 256)
    res_tasks<32, BF16>(task, ntask, rcv, B, ldb, C, ldc, P, ldp, col0, recs);
  else if (left >= 128)
    res_tasks<16, BF16>(task, ntask, rcv, B, ldb, C, ldc, P, ldp, col0, recs);
  else  // the last 64 columns
    res_tasks<8, BF16>(task, ntask, rcv, B, ldb, C, ldc, P, ldp, ldc - 64, recs);
}

// C row of a split row = the sum of its partial rows in a fixed order: a
// block takes FIN_COLS float4 columns of a row, and its thread groups every
// ng-th chunk each (group g: chunks g, g + ng, ...) before the group sums are
// added in group order.  A row of a few hundred chunks (a hub of a power-law
// graph) is then not one thread's serial chain of loads: with all of a row's
// columns in one block, four groups, the hubs of Chung-Lu 262144 took 15 us.
constexpr int FIN_THREADS = 256, FIN_COLS = 16;
__device__ __forceinline__ void add4(float4& s, const float4 x) {
  s.x += x.x;
  s.y += x.y;
  s.z += x.z;
  s.w += x.w;
}
__global__ void __launch_bounds__(FIN_THREADS)
    k_spmm_fin(const int4* __restrict__ multi, const float* __restrict__ P, int ldp, float* C, int ldc) {
  __shared__ float4 red[FIN_THREADS];
  const int cb = blockIdx.z * gridDim.y + blockIdx.y;  // column block (n is a multiple of 64: whole blocks)
  if (cb >= ldc / (4 * FIN_COLS)) return;
  const int4 m = multi[blockIdx.x];
  constexpr int ng = FIN_THREADS / FIN_COLS;
  const int g = threadIdx.x / FIN_COLS, qi = threadIdx.x % FIN_COLS;
  const int q = cb * FIN_COLS + qi;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  const float4* src = reinterpret_cast<const float4*>(P + (size_t)m.y * ldp) + q;
  const size_t row = ldp / 4, step = (size_t)ng * row;
  int j = g;
  for (; j + 3 * ng < m.z; j += 4 * ng) {  // four loads in flight, added in chunk order
    const float4* x = src + (size_t)j * row;
    const float4 x0 = x[0], x1 = x[step], x2 = x[2 * step], x3 = x[3 * step];
    add4(s, x0);
    add4(s, x1);
    add4(s, x2);
    add4(s, x3);
  }
  for (; j < m.z; j += ng) add4(s, src[(size_t)j * row]);
  red[threadIdx.x] = s;
  __syncthreads();
  if (g == 0) {
    const int used = m.z < ng ? m.z : ng;
    for (int h = 1; h < used; ++h) add4(s, red[h * FIN_COLS + qi]);
    reinterpret_cast<float4*>(C + (size_t)m.x * ldc)[q] = s;
  }
}

// The dense operand from features of another type or width: out (R x n, 16
// bits, row-major) = X (R x F, row stride ldx) rounded to nearest, columns F
// .. n - 1 zero; 8 columns a thread.  Bound by HBM: 65536 x 100 FP32 to 128
// FP16 columns 9 us.  vec: rows of X are 16-byte aligned.
template <class S, class D>
__global__ void __launch_bounds__(256)
    k_spmm_cast(const S* __restrict__ X, long long ldx, int R, int F, int n, bool vec, D* __restrict__ out) {
  const int nc = n / 8;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < (long long)R * nc;
       e += (long long)gridDim.x * blockDim.x) {
    const long long r = e / nc;
    const int c = (int)(e - r * nc) * 8;
    const S* src = X + r * ldx + c;
    alignas(16) S v[8];
    if (vec && c + 8 <= F) {
#pragma unroll
      for (int q = 0; q < (int)sizeof(v) / 16; ++q) reinterpret_cast<uint4*>(v)[q] = reinterpret_cast<const uint4*>(src)[q];
    } else {
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = c + q < F ? src[q] : S(0.f);
    }
    alignas(16) D o[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) o[q] = to_t<D>((float)v[q]);
    *reinterpret_cast<uint4*>(out + r * n + c) = *reinterpret_cast<const uint4*>(o);
  }
}

// ---------------------------------------------------------------------------
// Tensor-core kernel
// ---------------------------------------------------------------------------
struct SpmmArgs {
  const int4* part;        // work items {2 tile + add, first K-step, last + 1, partial slot or -1}
  const int* cols;
  const unsigned char* a;
  const unsigned char* B;  // dense operand, row-major, 16-bit values
  size_t ldb;              // its row stride in bytes
  const float* rscale;
  float* C;
  float* P;                // partial tiles of 128 rows, row stride ldc
  int R, n, ldc;
  int n256, n128;          // column blocks of 256 and of 128 columns; the others have 64
  uint32_t idesc[3];       // of 64, 128 and 256 columns
  int* err;
  uint32_t wait_limit;  // polls of a pipeline wait (copies <-> MMAs) before it gives up
};

// A stage holds KS K-steps (their A tiles, 4 KB each, come as one bulk copy)
// and is handed over once: a wait, a proxy fence, KS MMAs and a commit.  With
// a stage per K-step that chain of the issuing thread was the bound, 0.2 us a
// K-step at any width: a full V:2:8 operand (19456 rows) took 129 / 126 / 124
// us at n = 256 / 128 / 64; with the stages below 82 / 61 / 58 us, bound by
// the A tiles from HBM (378 MB, 6.2 TB/s at n = 128) and, at 256, by the
// 192 KB of copies in flight (4 producer warps: 143 us; stages of 2 K-steps:
// 126).
constexpr int SP_PF = 4;  // groups of stages whose column ids are loaded ahead (the ids come from DRAM)
constexpr int SP_PW = 8;  // producer warps

template <int NT, int KS, int ST>
struct SpmmSmem {
  static constexpr int B_BYTES = 16 * NT * 2;  // K=16 rows x NT columns, 16-bit
  alignas(1024) unsigned char b[ST][KS][B_BYTES];
  alignas(1024) unsigned char a[ST][KS * SP_KSTEP_BYTES];
  alignas(8) uint64_t full[ST];  // an arrival a producer lane, and the A copy's bytes
  alignas(8) uint64_t empty[ST];
  alignas(8) uint64_t done;
  int last_a;  // the last stage fill whose A copy was issued
  uint32_t tmem_base;
  int abort;
};

// One CTA: one work item (a tile, or a part of its K-steps) and NT columns
// of C.  The first SP_PW warps copy, each its share of the B rows of every
// stage, and read the accumulator out at the end; one lane of the last warp
// issues the MMAs.  That warp runs its loop whole, so that the descriptors
// stay in uniform registers (on one lane of a divergent branch an MMA took 85
// cycles to issue).
template <int NT, int KS, int ST>
__device__ __forceinline__ void spmm_item(const SpmmArgs& p, int n0, unsigned char* sp_raw) {
  static_assert(SP_THREADS == 32 * (SP_PW + 1), "the producer warps and the issuing warp");
  constexpr int WR = KS * 16 / SP_PW;  // a stage's B rows a producer warp
  using Smem = SpmmSmem<NT, KS, ST>;
  Smem& sm = *reinterpret_cast<Smem*>(
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(sp_raw) + 1023) & ~uintptr_t(1023)));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int4 item = p.part[blockIdx.x];
  const int t = item.x >> 1;
  const bool add = item.x & 1;  // the residual kernel wrote these rows first
  const uint32_t idesc = p.idesc[NT >> 7];  // (made here it cost 0.3 of 18 us: 4096 rows, V = 64, n = 128)
  const int s0 = item.y, nsteps = item.z - item.y;
  const int nst = (nsteps + KS - 1) / KS;  // stage fills
  ptx::grid_dependents_launch();

  if (tid == 0) {
    for (int s = 0; s < ST; ++s) {
      ptx::mbar_init(&sm.full[s], 32 * SP_PW + 1);
      ptx::mbar_init(&sm.empty[s], 1);
    }
    sm.last_a = -1;
    ptx::mbar_init(&sm.done, 1);
    sm.abort = 0;
    ptx::fence_mbar_init();
  }
  if (warp == 0) {
    ptx::tmem_alloc(&sm.tmem_base, NT);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = sm.tmem_base;

  int filled = 0;  // stage fills that this thread has arrived for
  if (warp < SP_PW) {
    // producer warps.  Lane l holds the column id of this warp's row l % WR
    // of the (l / WR)-th stage of each of the SP_PF groups of SG stages ahead
    // (issued well before use); every lane copies its 16-byte pieces of the
    // warp's B rows.
    constexpr int SG = 32 / WR;
    const uint64_t pol_a = ptx::policy_evict_first(), pol_b = ptx::policy_evict_last();
    auto ids = [&](int j) {  // group j
      const int k = (SG * j + lane / WR) * (KS * 16) + warp * WR + lane % WR;  // row of the item's operand
      return k < nsteps * 16 ? p.cols[(size_t)s0 * 16 + k] : -1;
    };
    int pf[SP_PF];
#pragma unroll
    for (int q = 0; q < SP_PF; ++q) pf[q] = ids(q);
    bool stop = false;
    for (int j = 0; SG * j < nst && !stop; ++j) {
      const int cur = pf[0];
#pragma unroll
      for (int q = 0; q + 1 < SP_PF; ++q) pf[q] = pf[q + 1];
      pf[SP_PF - 1] = ids(j + SP_PF);
      for (int d = 0; d < SG; ++d) {
        const int i = SG * j + d, s = i % ST;
        if (i >= nst) break;
        const bool ok = !*reinterpret_cast<volatile int*>(&sm.abort) &&
                        (i < ST || ptx::mbar_spin(&sm.empty[s], ((i / ST) - 1) & 1, p.wait_limit));
        if (!__all_sync(0xffffffffu, ok)) {
          if (lane == 0) {
            atomicOr(p.err, 1);
            sm.abort = 1;
          }
          stop = true;
          break;
        }
        ++filled;
        if (warp == 0 && lane == 0) {
          // A tiles are read once: evict-first, so that they do not push
          // the B rows (read by every tile) out of L2
          const uint32_t bytes = (uint32_t)min(KS, nsteps - i * KS) * SP_KSTEP_BYTES;
          sm.last_a = i;
          ptx::mbar_arrive_expect_tx(&sm.full[s], bytes);
          ptx::bulk_g2s_hint(sm.a[s], p.a + (size_t)(s0 + i * KS) * SP_KSTEP_BYTES, bytes, &sm.full[s], pol_a);
        }
        // the 16 B rows: each lane copies 16-byte chunks into the
        // 128-byte-swizzled layout of the MMA's B operand (atoms of 8 k-rows
        // x 128 bytes, n-atoms 2048 bytes apart, k-atoms 1024 bytes apart,
        // chunk j of k-row r stored at chunk j ^ (r % 8))
        // (rows past the item's last K-step land in places no MMA reads)
        {
          constexpr int CPR = NT / 8;                      // 16-byte chunks per row
          constexpr int RPI = 32 / CPR;                    // rows per warp instruction
          const int c = lane % CPR, sub = lane / CPR;
          unsigned char* bs = &sm.b[s][0][0];
          const unsigned char* bcol = p.B + (size_t)(n0 + 8 * c) * 2;
#pragma unroll
          for (int r0 = 0; r0 < WR; r0 += RPI) {
            const int k = warp * WR + r0 + sub, kr = k % 16;  // row of the stage, of its K-step
            const int row = __shfl_sync(0xffffffffu, cur, d * WR + r0 + sub);
            // a padding column (-1): its A column is zero; fill zeros, read nothing
            const unsigned char* src = bcol + (size_t)(row < 0 ? 0 : row) * p.ldb;
            unsigned char* dst = bs + (k / 16) * Smem::B_BYTES + (c >> 3) * 2048 + (kr >> 3) * 1024 + (kr & 7) * 128 +
                                 (((c & 7) ^ (kr & 7)) << 4);
            ptx::cp_async16_zfill_hint(dst, src, row < 0 ? 0u : 16u, pol_b);
          }
        }
        ptx::cp_async_mbar_arrive(&sm.full[s]);
        __syncwarp();
      }
    }
    if (stop) ptx::cp_async_wait_all();  // nothing of this thread's is in flight when the CTA leaves
  } else {
    const bool leader = ptx::elect_one();
    for (int i = 0; i < nst; ++i) {
      const int s = i % ST;
      const bool ok = ptx::mbar_spin(&sm.full[s], (i / ST) & 1, p.wait_limit);
      if (!__all_sync(0xffffffffu, ok)) {
        if (leader) {
          atomicOr(p.err, 2);
          sm.abort = 1;
        }
        break;
      }
      // the B rows were written by the load/store path: order them before
      // the tensor core reads shared memory
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      ptx::tc_fence_after();
      const uint64_t adesc = ptx::smem_desc(ptx::smem_addr(sm.a[s]), 128, 256, 0);
      const uint64_t bdesc = ptx::smem_desc(ptx::smem_addr(sm.b[s]), 2048, 1024, 2);
      const int ks = min(KS, nsteps - i * KS);
      if (leader) {
#pragma unroll
        for (int k = 0; k < KS; ++k)
          if (k < ks)
            ptx::mma_f16(tmem, adesc + (uint64_t)(k * (SP_KSTEP_BYTES >> 4)),
                         bdesc + (uint64_t)(k * (Smem::B_BYTES >> 4)), idesc, (i | k) > 0 ? 1u : 0u);
        ptx::mma_commit(&sm.empty[s]);
      }
    }
    if (leader) ptx::mma_commit(&sm.done);
  }
  __syncwarp();
  // everybody waits for the last MMA
  bool ok = ptx::mbar_wait(&sm.done, 0, SP_WAIT_LIMIT);
  if (!ok && tid == 0) atomicOr(p.err, 4);
  __syncthreads();
  if (sm.abort || !ok) {
    // a wait gave up: before the CTA leaves, every A copy lands.  The
    // producers that stopped early arrive for the fills they missed (at most
    // one a stage, as a stage is filled again only after it was used), which
    // completes the phase of each stage's last fill.
    if (warp < SP_PW)
      for (int i = filled; i <= sm.last_a; ++i) ptx::mbar_arrive(&sm.full[i % ST]);
    if (tid == 0)
      for (int i = max(sm.last_a - ST + 1, 0); i <= sm.last_a; ++i)
        ptx::mbar_wait(&sm.full[i % ST], (i / ST) & 1, SP_WAIT_LIMIT);
  }
  __syncthreads();
  ptx::tc_fence_after();
  if (ok && !sm.abort && warp < SP_PW) {
    // warp w reads TMEM lanes 32 (w % 4) .. of half of the columns; a part of
    // a split tile goes out as it is,
    // through a 32 x 32 piece of shared memory (the stages are free now), so
    // that a warp reads and writes whole 128-byte lines of C
    constexpr int CW = NT / (SP_PW / 4), EP = 36;
    static_assert(sizeof(sm.b) + sizeof(sm.a) >= SP_PW * 32 * EP * sizeof(float), "the pieces fit the stages");
    float* piece = reinterpret_cast<float*>(&sm.b[0][0][0]) + warp * (32 * EP);
    const bool whole = item.w < 0;
    const int r0 = (warp & 3) * 32, row0 = t * SP_TM + r0;  // the warp's first row of the tile, of C
    const float sc = whole ? (row0 + lane < p.R ? p.rscale[row0 + lane] : 0.f) : 1.f;
    const int live = whole ? p.R - row0 : 32;  // rows of the warp that are written
    float* out = whole ? p.C + (size_t)row0 * p.ldc : p.P + ((size_t)item.w * SP_TM + r0) * p.ldc;
    out += (size_t)(lane >> 3) * p.ldc + n0 + (lane & 7) * 4;
#pragma unroll 1
    for (int c0 = (warp >> 2) * CW; c0 < (warp >> 2) * CW + CW; c0 += 32) {
      float4 was[8];
      if (whole && add) {
#pragma unroll
        for (int q = 0; q < 8; ++q)
          if (4 * q + (lane >> 3) < live) was[q] = *reinterpret_cast<const float4*>(out + (size_t)(4 * q) * p.ldc + c0);
      }
      uint32_t v[32];
      ptx::tmem_ld_32x32b_x32(tmem + ((uint32_t)r0 << 16) + (uint32_t)c0, v);
      ptx::tmem_ld_wait();
#pragma unroll
      for (int q = 0; q < 8; ++q)
        *reinterpret_cast<float4*>(piece + lane * EP + 4 * q) =
            make_float4(__uint_as_float(v[4 * q]) * sc, __uint_as_float(v[4 * q + 1]) * sc,
                        __uint_as_float(v[4 * q + 2]) * sc, __uint_as_float(v[4 * q + 3]) * sc);
      __syncwarp();
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        float4 o = *reinterpret_cast<const float4*>(piece + (4 * q + (lane >> 3)) * EP + (lane & 7) * 4);
        if (whole && add) add4(o, was[q]);
        if (4 * q + (lane >> 3) < live) *reinterpret_cast<float4*>(out + (size_t)(4 * q) * p.ldc + c0) = o;
      }
      __syncwarp();
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 0) ptx::tmem_dealloc(tmem, NT);
}

// Stages of each width: 192 KB of copies in flight.
using SpmmSmem256 = SpmmSmem<256, 4, 4>;
using SpmmSmem128 = SpmmSmem<128, 8, 3>;
using SpmmSmem64 = SpmmSmem<64, 8, 4>;
// W: the width of all column blocks, or 0 for several (a product of 2048 rows,
// V:2:8, n = 64 takes 7.0 us, with the width chosen in the kernel 7.2).
template <int W>
__global__ void __launch_bounds__(SP_THREADS, 1) k_spmm_vnm(const __grid_constant__ SpmmArgs p) {
  extern __shared__ unsigned char sp_raw[];
  const int y = blockIdx.y, y128 = W == 256 ? -1 : W ? y : y - p.n256, y64 = W == 128 ? -1 : W ? y : y128 - p.n128;
  if (y128 < 0) spmm_item<256, 4, 4>(p, 256 * y, sp_raw);
  else if (y64 < 0) spmm_item<128, 8, 3>(p, W ? 128 * y : 256 * p.n256 + 128 * y128, sp_raw);
  else spmm_item<64, 8, 4>(p, W ? 64 * y : 256 * p.n256 + 128 * p.n128 + 64 * y64, sp_raw);
}

// Rows of a split tile: the sum of its parts in order, scaled, added to what
// the residual kernel wrote.  Bound by L2 (the parts were just written): one
// float4 of C a thread, the parts' loads eight in flight.  (P is written while
// this kernel is set up already, so it is not __restrict__: loads of memory that
// is constant for a kernel's life may be made before the wait.)
__global__ void __launch_bounds__(256)
    k_spmm_tfin(const int4* __restrict__ split, const float* P, const float* __restrict__ rscale, int R, int n,
                float* __restrict__ C) {
  ptx::grid_dependency_wait();
  const int4 m = split[blockIdx.x];
  const int t = m.x >> 1, nq = n / 4;
  const int e = (blockIdx.z * gridDim.y + blockIdx.y) * blockDim.x + threadIdx.x, rt = e / nq, q = e % nq;
  const int row = t * SP_TM + rt;
  if (rt >= SP_TM || row >= R) return;
  {
    const float4* src = reinterpret_cast<const float4*>(P + ((size_t)m.y * SP_TM + rt) * n) + q;
    const size_t step = (size_t)SP_TM * nq;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int k = 0; k < m.z; ++k) add4(s, src[k * step]);
    const float sc = rscale[row];
    float4 o = make_float4(s.x * sc, s.y * sc, s.z * sc, s.w * sc);
    float4* dst = reinterpret_cast<float4*>(C + (size_t)row * n) + q;
    if (m.x & 1) add4(o, *dst);
    *dst = o;
  }
}

// ---------------------------------------------------------------------------
// Host
// ---------------------------------------------------------------------------
static int spmm_dense_min(int V) {
  if (const char* e = getenv("VNM_SPMM_DENSE_MIN")) {
    const int v = atoi(e);
    if (v >= 0) return v;
  }
  return V;
}

// Poll limit of the tensor kernel's pipeline waits.  A test hook,
// VNM_SPMM_TEST_WAIT_LIMIT, sets a small one so that a wait runs out and the
// kernel takes its error path (stop issuing, let the copies in flight land,
// report); the wait for the last MMA and the drain keep the full limit.
static uint32_t spmm_wait_limit() {
  if (const char* e = getenv("VNM_SPMM_TEST_WAIT_LIMIT")) {
    const long v = atol(e);
    if (v > 0) return (uint32_t)v;
  }
  return SP_SPIN_LIMIT;
}

// Arena bytes compress_t takes for nnz entries and R rows.
static size_t compress_scratch_bytes(int R, int nnz) {
  const int ntiles = (R + SP_TM - 1) / SP_TM;
  const size_t n = nnz > 0 ? (size_t)nnz : 1;
  size_t b = arena_bytes(n, 8) + 3 * arena_bytes(n, 4);  // keys, dlist, gofs, rpos
  b += 2 * arena_bytes(n, 4) + 2 * arena_bytes(ntiles + 1, 4) + 2 * arena_bytes((size_t)R + 2, 4) +
       arena_bytes(CC_N, 4);                             // zeroed: gsl, resflag, tile_raw, tile_res, rowlen, bmax, counters
  b += arena_bytes(n, 8) + arena_bytes(n, 4);            // residual keys and sources
  b += 2 * radix_sort_scratch_bytes(nnz);
  b += 2 * arena_bytes(ntiles + 1, 4) + arena_bytes(ntiles + 1, 16);  // tile_base, tile_rawbase, tile_plan
  b += arena_bytes(R / RP_TILE + 1, 16);                              // sums
  b += 2 * scan_scratch_bytes((nnz > R ? nnz : R) + 1) + 16384;
  return b;
}

template <class T>
static vnm_status compress_t(vnm_ctx* ctx, int R, int nnz, const int* d_row, const int* d_col, const float* d_val,
                             int M, int V, vnm_spmm_matrix* out) {
  const int nseg = (R + M - 1) / M;
  const int nbrow = (R + V - 1) / V;
  const int ntiles = (R + SP_TM - 1) / SP_TM;
  const int rtiles = (R + RP_TILE - 1) / RP_TILE;
  const int dense_min = spmm_dense_min(V);
  const int bm = key_bits_m(M), bv = __builtin_ctz((unsigned)V), sh = bm + bv;  // V is a power of two (divides 128)
  int* h = ctx->h_pinned;
  const size_t n1 = nnz > 0 ? (size_t)nnz : 1;
  unsigned long long* keys = arena_take<unsigned long long>(ctx, n1);
  int* dlist = arena_take<int>(ctx, n1);
  int* gofs = arena_take<int>(ctx, n1);
  int* rpos = arena_take<int>(ctx, n1);
  int* tile_base = arena_take<int>(ctx, ntiles + 1);
  int* tile_rawbase = arena_take<int>(ctx, ntiles + 1);
  int4* tile_plan = arena_take<int4>(ctx, ntiles + 1);
  int* sums = arena_take<int>(ctx, rtiles);
  const size_t zero0 = ctx->arena.used;  // zeroed together from here
  int* gsl = arena_take<int>(ctx, n1);
  int* resflag = arena_take<int>(ctx, n1);
  int* tile_raw = arena_take<int>(ctx, ntiles + 1);
  int* tile_res = arena_take<int>(ctx, ntiles + 1);
  int* rowlen = arena_take<int>(ctx, (size_t)R + 1);
  unsigned* bmax = arena_take<unsigned>(ctx, nbrow + 1);
  int* counters = arena_take<int>(ctx, CC_N);
  if (!keys || !dlist || !gofs || !rpos || !tile_base || !tile_rawbase || !tile_plan || !sums || !gsl || !resflag ||
      !tile_raw || !tile_res || !rowlen || !bmax || !counters)
    return VNM_ERR_NOMEM;
  cudaStream_t st = ctx->stream;
  VNM_CUDA_TRY(cudaMemsetAsync(ctx->arena.base + zero0, 0, ctx->arena.used - zero0, st));
  unsigned long long* skeys = keys;
  int* spos = nullptr;
  if (nnz > 0) {
    VNM_LAUNCH(ctx, k_cmp_keys, sp_grid(ctx, nnz), 256, 0, d_row, d_col, d_val, nnz, M, V, nseg, bm, bv, keys, bmax,
               counters + CC_UNSORTED);
    const long long maxkey = ((long long)nbrow * nseg) << sh;
    VNM_TRY(radix_sort_u64(ctx, keys, nullptr, nnz, sp_bits(maxkey), &skeys, &spos));
    VNM_LAUNCH(ctx, k_cmp_groups, sp_grid(ctx, nnz), 256, 0, skeys, spos, nnz, V, nseg, bm, dense_min, dlist, resflag,
               rowlen, tile_res, counters);
    // the number of dense blocks stays on the device until the storage is sized
    VNM_LAUNCH(ctx, k_cmp_dense, sp_grid(ctx, nnz, DB_WARPS * 32), DB_WARPS * 32, 0, skeys, dlist, nnz, V, nseg, bm,
               gsl, tile_raw, counters);
  }
  VNM_LAUNCH(ctx, k_tile_plan, 1, 1024, 0, tile_raw, ntiles, ctx->num_sms, tile_base, tile_rawbase, tile_plan,
             counters);
  VNM_LAUNCH(ctx, k_res_plan, rtiles, RP_TILE, 0, rowlen, R, tile_raw, tile_res, sums, counters);
  VNM_CUDA_TRY(cudaMemcpyAsync(h, counters, CC_N * sizeof(int), cudaMemcpyDeviceToHost, st));
  VNM_CUDA_TRY(cudaStreamSynchronize(st));
  const int padded = h[CC_PADDED], ngroups = h[CC_GROUPS], nd = h[CC_DENSE];
  const bool unsorted = h[CC_UNSORTED] != 0;
  out->npart = h[CC_PARTS];
  out->ntsplit = h[CC_SPLIT];
  out->ntslots = h[CC_SLOTS];
  out->valid_blocks = h[CC_VALID];
  out->slices = h[CC_SLICES];
  out->ntt = h[CC_TILES];
  out->nres = h[CC_RES];
  out->nslots = h[CC_CLASS];
  out->ntask = 0;
  for (int k = 0; k < TASK_CLASSES; ++k) out->ntask += h[CC_CLASS + k];
  out->nmulti = h[CC_MULTI_ROWS];
  out->dense_min = dense_min;
  out->slices_padded = padded;
  out->groups = ngroups;
  out->nsteps = padded / 4;
  out->ntiles = ntiles;
  // the matrix's own storage (kept across calls)
  const size_t b_pt = arena_bytes((size_t)out->npart + 1, 16), b_ts = arena_bytes((size_t)out->ntsplit + 1, 16),
               b_cols = arena_bytes((size_t)out->nsteps * 16 + 1, 4),
               b_a = arena_bytes((size_t)out->nsteps * SP_KSTEP_BYTES + 16, 1),
               b_sc = arena_bytes((size_t)ntiles * SP_TM, 4), b_rc = arena_bytes((size_t)out->nres + 1, 8),
               b_tk = arena_bytes((size_t)out->ntask + 1, 16),
               b_mu = arena_bytes((size_t)out->nmulti + 1, 16);
  // with room for the asynchronous entry point's flag and partial sums up to
  // PART_COLS columns, so that a first product allocates nothing
  size_t pfloats = ((size_t)out->nslots + (size_t)out->ntslots * SP_TM) * PART_COLS + 1;
  if (pfloats * sizeof(float) > PART_BYTES_MAX) pfloats = 1;
  const size_t b_err = arena_bytes(1, 4), b_part = arena_bytes(pfloats, 4);
  const size_t need = b_pt + b_ts + b_cols + b_a + b_sc + b_rc + b_tk + b_mu + b_err + b_part;
  void* base = nullptr;
  size_t have = 0;
  bool pending = false;
  if (ctx->spare) {  // a freed operand's storage, when large enough
    std::lock_guard<std::mutex> g(ctx->spare->m);
    if (ctx->spare->ptr && ctx->spare->bytes >= need) {
      base = ctx->spare->ptr;
      have = ctx->spare->bytes;
      pending = ctx->spare->pending;
      ctx->spare->ptr = nullptr;
      ctx->spare->bytes = 0;
    }
  }
  if (!base) {
    VNM_CUDA_TRY(cudaMalloc(&base, need));
    have = need;
  }
  out->base = base;
  out->bytes = have;
  // The freed operand's asynchronous products run on its caller's streams,
  // possibly from a captured graph, and read and write this storage: they end
  // before anything is written to it.  (The wait is here and not in the free,
  // which a training loop calls beside its running products.)
  if (pending) VNM_CUDA_TRY(cudaDeviceSynchronize());
  char* pb = static_cast<char*>(base);
  size_t o = 0;
  out->part_list = reinterpret_cast<int4*>(pb + o);
  o += b_pt;
  out->tsplit = reinterpret_cast<int4*>(pb + o);
  o += b_ts;
  out->cols = reinterpret_cast<int*>(pb + o);
  o += b_cols;
  out->a = reinterpret_cast<unsigned char*>(pb + o);
  o += b_a;
  out->rscale = reinterpret_cast<float*>(pb + o);
  o += b_sc;
  out->rcv = reinterpret_cast<int2*>(pb + o);
  o += b_rc;
  out->task = reinterpret_cast<int4*>(pb + o);
  o += b_tk;
  out->multi = reinterpret_cast<int4*>(pb + o);
  o += b_mu;
  out->err = reinterpret_cast<int*>(pb + o);
  o += b_err;
  out->part = reinterpret_cast<float*>(pb + o);
  out->part_floats = pfloats;
  VNM_CUDA_TRY(cudaMemsetAsync(out->err, 0, sizeof(int), st));
  // residual CSR: the residual entries in their original order, stably
  // sorted by row (which they are when the rows never decrease)
  if (out->nres > 0) {
    VNM_TRY(exclusive_scan(ctx, resflag, rpos, nnz, nullptr));
    if (!unsorted) {
      VNM_LAUNCH(ctx, k_res_sorted, sp_grid(ctx, nnz), 256, 0, resflag, rpos, d_col, d_val, nnz, out->rcv);
    } else {
      unsigned long long* rkey = arena_take<unsigned long long>(ctx, (size_t)out->nres);
      int* rsrc = arena_take<int>(ctx, (size_t)out->nres);
      if (!rkey || !rsrc) return VNM_ERR_NOMEM;
      VNM_LAUNCH(ctx, k_res_compact, sp_grid(ctx, nnz), 256, 0, resflag, rpos, d_row, nnz, rkey, rsrc);
      unsigned long long* sk = nullptr;
      int* ss = nullptr;
      VNM_TRY(radix_sort_u64(ctx, rkey, rsrc, (int)out->nres, sp_bits(R), &sk, &ss));
      VNM_LAUNCH(ctx, k_res_gather, sp_grid(ctx, out->nres), 256, 0, ss, d_col, d_val, (int)out->nres, out->rcv);
    }
  }
  if (out->ntask > 0)
    VNM_LAUNCH(ctx, k_res_tasks, rtiles, RP_TILE, 0, rowlen, R, tile_raw, tile_res, sums, counters, out->task,
               out->multi);
  if (out->ntt > 0)
    VNM_LAUNCH(ctx, k_tile_parts, sp_grid(ctx, ntiles), 256, 0, tile_raw, tile_res, ntiles, tile_base, tile_plan,
               out->part_list, out->tsplit);
  if (nd > 0) {
    VNM_CUDA_TRY(cudaMemsetAsync(out->cols, 0xff, b_cols, st));  // -1: padding columns
    VNM_CUDA_TRY(cudaMemsetAsync(out->a, 0, b_a, st));
    VNM_TRY(exclusive_scan(ctx, gsl, gofs, nnz, nullptr));
    VNM_LAUNCH(ctx, k_cmp_fill<T>, sp_grid(ctx, nd, DB_WARPS), DB_WARPS * 32, 0, skeys, spos, d_val, dlist, nd, nnz, M,
               V, nseg, bm, gofs, tile_base, tile_rawbase, bmax, out->cols, out->a);
  }
  VNM_LAUNCH(ctx, k_cmp_rscale, sp_grid(ctx, (long long)ntiles * SP_TM), 256, 0, bmax, ntiles, R, V, out->rscale);
  return VNM_OK;
}

// x by `blocks` blocks, in y and, past what y holds, z (blocks may be a few more).
static dim3 grid_yz(int x, int blocks) {
  const int z = (blocks + 65534) / 65535;
  return dim3((unsigned)x, (unsigned)((blocks + z - 1) / z), (unsigned)z);
}

// One launch for all column blocks (n256 of 256 columns, n128 of 128, n64 of
// 64): for the same reason as the residual kernel's, and so that no width
// waits for another's last tiles.
static vnm_status launch_spmm(vnm_ctx* ctx, const vnm_spmm_matrix* A, SpmmArgs& p, int n256, int n128, int n64) {
  constexpr size_t smem =
      std::max({sizeof(SpmmSmem256), sizeof(SpmmSmem128), sizeof(SpmmSmem64)}) + 1024;
  // one CTA an SM: its accumulator's tensor-memory columns are always free
  static_assert(2 * smem > (228u << 10), "an allocation never waits for another CTA");
  p.n256 = n256;
  p.n128 = n128;
  for (int k = 0; k < 3; ++k) p.idesc[k] = ptx::idesc_f16(A->dtype == 1 ? 1u : 0u, 0u, 1u, SP_TM, 64u << k);
  const auto kernel = n128 + n64 == 0    ? k_spmm_vnm<256>
                      : n256 + n64 == 0  ? k_spmm_vnm<128>
                      : n256 + n128 == 0 ? k_spmm_vnm<64>
                                         : k_spmm_vnm<0>;
  VNM_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  VNM_LAUNCH(ctx, kernel, dim3(A->npart, n256 + n128 + n64), SP_THREADS, smem, p);
  return VNM_OK;
}

}  // namespace vnm

using namespace vnm;

extern "C" {

vnm_status vnm_spmm_compress(vnm_ctx* ctx, int nrows, int nnz, const int* row, const int* col, const float* val,
                             int mem, int M, int V, int dtype, vnm_spmm_matrix** out) {
  if (!ctx || !out || nrows <= 0 || nnz < 0 || M < 2 || M > 8 || V < 1 || (SP_TM % V) != 0) return VNM_ERR_ARG;
  if (dtype != 0 && dtype != 1) return VNM_ERR_ARG;
  if (mem != VNM_MEM_HOST && mem != VNM_MEM_DEVICE) return VNM_ERR_ARG;
  if (nnz > 0 && (!row || !col || !val)) return VNM_ERR_ARG;
  *out = nullptr;
  const size_t need = 3 * arena_bytes(nnz, 4) + compress_scratch_bytes(nrows, nnz);
  VNM_TRY(arena_reserve(ctx, need));
  VNM_TRY(pinned_reserve(ctx, 64));
  VNM_TRY(begin_call(ctx));
  const int *d_row, *d_col;
  const float* d_val;
  VNM_TRY(stage_in(ctx, row, nnz, mem, &d_row));
  VNM_TRY(stage_in(ctx, col, nnz, mem, &d_col));
  VNM_TRY(stage_in(ctx, val, nnz, mem, &d_val));
  vnm_spmm_matrix* A = new vnm_spmm_matrix();
  A->device = ctx->device;
  A->R = nrows;
  A->M = M;
  A->V = V;
  A->dtype = dtype;
  A->nnz = nnz;
  vnm_status st = dtype == 1 ? compress_t<__nv_bfloat16>(ctx, nrows, nnz, d_row, d_col, d_val, M, V, A)
                             : compress_t<__half>(ctx, nrows, nnz, d_row, d_col, d_val, M, V, A);
  if (st == VNM_OK) st = end_call(ctx);
  if (st != VNM_OK) {
    if (A->base) cudaFree(A->base);
    delete A;
    return st;
  }
  if (ctx->spare) {
    std::lock_guard<std::mutex> g(ctx->spare->m);
    ctx->spare->refs++;
    A->spare = ctx->spare;
  }
  *out = A;
  return VNM_OK;
}

vnm_status vnm_spmm_info(const vnm_spmm_matrix* A, long long* info, int n) {
  if (!A || !info) return VNM_ERR_ARG;
  const long long v[13] = {A->nnz, A->groups, A->valid_blocks, A->slices, A->slices_padded, A->nsteps, A->ntiles,
                           (long long)A->nsteps * SP_KSTEP_BYTES, A->nres, A->ntask, A->ntt, A->dense_min,
                           A->nslots};
  for (int i = 0; i < n && i < 13; ++i) info[i] = v[i];
  return VNM_OK;
}

vnm_status vnm_spmm_free(vnm_spmm_matrix* A) {
  if (!A) return VNM_ERR_ARG;
  cudaSetDevice(A->device);
  if (A->part_own) cudaFree(A->part);
  bool last = false;
  if (A->spare) {
    // keep the storage for the context's next compression (the larger of
    // this block and the one kept, while the context lives)
    std::lock_guard<std::mutex> g(A->spare->m);
    if (A->base && A->spare->ctx_alive && A->bytes > A->spare->bytes) {
      if (A->spare->ptr) cudaFree(A->spare->ptr);
      A->spare->ptr = A->base;
      A->spare->bytes = A->bytes;
      A->spare->pending = A->pending;
      A->base = nullptr;
    }
    last = --A->spare->refs == 0;
  }
  if (A->base) cudaFree(A->base);
  if (last) delete A->spare;
  delete A;
  return VNM_OK;
}

// Enqueue one product on ctx->stream: the residual kernels, then the tensor
// kernel and the sum of its split tiles.  dB, dC, P and err are device memory.
static vnm_status spmm_enqueue(vnm_ctx* ctx, const vnm_spmm_matrix* A, const void* dB, int n, float* dC, float* P,
                               int* err, bool timed) {
  SpmmArgs p;
  p.part = A->part_list;
  p.cols = A->cols;
  p.a = A->a;
  p.B = static_cast<const unsigned char*>(dB);
  p.ldb = (size_t)n * 2;
  p.rscale = A->rscale;
  p.C = dC;
  p.P = P + (size_t)A->nslots * n;  // after the residual's partial rows
  p.R = A->R;
  p.n = n;
  p.ldc = n;
  p.err = err;
  p.wait_limit = spmm_wait_limit();
  // the CUDA-core part: 8 columns a lane
  auto launch_res = [&]() -> vnm_status {
    if (A->ntask > 0) {
      // one wave of resident blocks (the task list is walked with a stride)
      const int per_block = RES_THREADS / 32;
      int bx = (A->ntask + per_block - 1) / per_block;
      if (bx > ctx->num_sms * RES_BLOCKS_PER_SM) bx = ctx->num_sms * RES_BLOCKS_PER_SM;
      const dim3 grid((unsigned)bx, (unsigned)col_blocks(n));
      if (A->dtype == 1)
        VNM_LAUNCH(ctx, k_spmm_res<true>, grid, RES_THREADS, 0, A->task, A->ntask, A->rcv, p.B, (unsigned)p.ldb, dC, n,
                   P, n);
      else
        VNM_LAUNCH(ctx, k_spmm_res<false>, grid, RES_THREADS, 0, A->task, A->ntask, A->rcv, p.B, (unsigned)p.ldb, dC, n,
                   P, n);
    }
    if (A->nmulti > 0)
      VNM_LAUNCH(ctx, k_spmm_fin, grid_yz(A->nmulti, n / (4 * FIN_COLS)), FIN_THREADS, 0, A->multi, P, n, dC, n);
    return VNM_OK;
  };
  // The operand is read once a column block: n = 192 as 128 + 64 instead of
  // three times 64.  VNM_SPMM_WIDTH (64, 128 or 256) in the environment fixes the
  // tensor kernel's width where it divides n.
  int fixed = 0;
  if (const char* e = getenv("VNM_SPMM_WIDTH")) {
    const int w = atoi(e);
    if ((w == 64 || w == 128 || w == 256) && n % w == 0) fixed = w;
  }
  auto launch_nt = [&]() -> vnm_status {
    if (A->ntt == 0) return VNM_OK;
    const int n256 = fixed == 256 ? n / 256 : fixed ? 0 : n / 256;
    const int n128 = fixed == 128 ? n / 128 : fixed ? 0 : (n % 256) / 128;
    const int n64 = fixed == 64 ? n / 64 : fixed ? 0 : (n % 128) / 64;
    VNM_TRY(launch_spmm(ctx, A, p, n256, n128, n64));
    if (A->ntsplit == 0) return VNM_OK;
    cudaLaunchAttribute attr[1];  // set up while the parts are made
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.stream = ctx->stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.gridDim = grid_yz(A->ntsplit, SP_TM * (n / 4) / 256);
    cfg.blockDim = dim3(256);
    VNM_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_spmm_tfin, (const int4*)A->tsplit, (const float*)p.P,
                                    (const float*)A->rscale, A->R, n, dC));
    ctx->launches++;
    return VNM_OK;
  };
  if (timed) VNM_CUDA_TRY(cudaEventRecord(ctx->ev_main0, ctx->stream));
  VNM_TRY(launch_res());
  VNM_TRY(launch_nt());
  if (timed) VNM_CUDA_TRY(cudaEventRecord(ctx->ev_main1, ctx->stream));
  return VNM_OK;
}

vnm_status vnm_spmm_run(vnm_ctx* ctx, const vnm_spmm_matrix* A, const void* B, int n, float* C, int mem) {
  if (!ctx || !A || !B || !C || n <= 0 || (n % 64) != 0) return VNM_ERR_ARG;
  if (mem != VNM_MEM_HOST && mem != VNM_MEM_DEVICE) return VNM_ERR_ARG;
  if (A->device != ctx->device) return VNM_ERR_ARG;
  const size_t bbytes = (size_t)A->R * n * 2, cbytes = (size_t)A->R * n * sizeof(float);
  const size_t pfloats = ((size_t)A->nslots + (size_t)A->ntslots * SP_TM) * n + 1;
  const size_t pbytes = arena_bytes(pfloats, sizeof(float));
  VNM_TRY(arena_reserve(ctx, (mem == VNM_MEM_HOST ? bbytes + cbytes + 512 : 0) + pbytes + 4096));
  VNM_TRY(pinned_reserve(ctx, 64));
  VNM_TRY(begin_call(ctx));
  const void* dB = B;
  float* dC = C;
  if (mem == VNM_MEM_HOST) {
    void* tb = arena_take<unsigned char>(ctx, bbytes);
    dC = arena_take<float>(ctx, (size_t)A->R * n);
    if (!tb || !dC) return VNM_ERR_NOMEM;
    VNM_CUDA_TRY(cudaMemcpyAsync(tb, B, bbytes, cudaMemcpyHostToDevice, ctx->stream));
    dB = tb;
  }
  if ((reinterpret_cast<uintptr_t>(dB) & 15) != 0 || (reinterpret_cast<uintptr_t>(dC) & 15) != 0)
    return VNM_ERR_ARG;
  float* P = arena_take<float>(ctx, pfloats);
  int* err = arena_take<int>(ctx, 1);
  if (!err || !P) return VNM_ERR_NOMEM;
  VNM_CUDA_TRY(cudaMemsetAsync(err, 0, sizeof(int), ctx->stream));
  VNM_TRY(spmm_enqueue(ctx, A, dB, n, dC, P, err, true));
  VNM_CUDA_TRY(cudaMemcpyAsync(ctx->h_pinned, err, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  if (mem == VNM_MEM_HOST)
    VNM_CUDA_TRY(cudaMemcpyAsync(C, dC, cbytes, cudaMemcpyDeviceToHost, ctx->stream));
  VNM_TRY(end_call(ctx));
  VNM_CUDA_TRY(cudaEventElapsedTime(&ctx->main_ms, ctx->ev_main0, ctx->ev_main1));
  if (ctx->h_pinned[0] != 0) return VNM_ERR_INTERNAL;
  return VNM_OK;
}

vnm_status vnm_spmm_run_async(vnm_ctx* ctx, vnm_spmm_matrix* A, const void* B, int n, float* C, void* stream) {
  if (!ctx || !A || !B || !C || n <= 0 || (n % 64) != 0) return VNM_ERR_ARG;
  if (A->device != ctx->device) return VNM_ERR_ARG;
  if ((reinterpret_cast<uintptr_t>(B) & 15) != 0 || (reinterpret_cast<uintptr_t>(C) & 15) != 0) return VNM_ERR_ARG;
  VNM_CUDA_TRY(cudaSetDevice(ctx->device));
  const size_t need = ((size_t)A->nslots + (size_t)A->ntslots * SP_TM) * n + 1;
  if (need > A->part_floats) {  // the first call for a larger n: make room (this waits for the device)
    if (A->part_own) VNM_CUDA_TRY(cudaFree(A->part));
    A->part = nullptr;
    A->part_floats = 0;
    A->part_own = false;
    VNM_CUDA_TRY(cudaMalloc(&A->part, need * sizeof(float)));
    A->part_floats = need;
    A->part_own = true;
  }
  ctx->launches = 0;
  ctx->last_ms = ctx->main_ms = 0.f;
  cudaStream_t own = ctx->stream;
  ctx->stream = static_cast<cudaStream_t>(stream);
  A->pending = true;
  const vnm_status st = spmm_enqueue(ctx, A, B, n, C, A->part, A->err, false);
  ctx->stream = own;
  return st;
}

vnm_status vnm_spmm_run_cast_async(vnm_ctx* ctx, vnm_spmm_matrix* A, const void* X, int xtype, long long ldx, int F,
                                   void* B, int n, float* C, void* stream) {
  if (!ctx || !A || !X || !B || !C || xtype < 0 || xtype > 2 || F <= 0 || ldx < F || n < F || (n % 64) != 0)
    return VNM_ERR_ARG;
  const size_t xsize = xtype == 2 ? 4 : 2;
  if (A->device != ctx->device || reinterpret_cast<uintptr_t>(X) % xsize != 0 ||
      (reinterpret_cast<uintptr_t>(B) & 15) != 0 || (reinterpret_cast<uintptr_t>(C) & 15) != 0)
    return VNM_ERR_ARG;
  VNM_CUDA_TRY(cudaSetDevice(ctx->device));
  const bool vec = (reinterpret_cast<uintptr_t>(X) & 15) == 0 && (ldx * xsize) % 16 == 0;
  long long g = ((long long)A->R * (n / 8) + 255) / 256;
  if (g > (long long)ctx->num_sms * 32) g = (long long)ctx->num_sms * 32;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
#define VNM_CAST(S)                                                                                              \
  do {                                                                                                           \
    if (A->dtype == 1)                                                                                           \
      k_spmm_cast<S, __nv_bfloat16><<<(unsigned)g, 256, 0, st>>>(static_cast<const S*>(X), ldx, A->R, F, n, vec, \
                                                                 static_cast<__nv_bfloat16*>(B));                \
    else                                                                                                         \
      k_spmm_cast<S, __half><<<(unsigned)g, 256, 0, st>>>(static_cast<const S*>(X), ldx, A->R, F, n, vec,        \
                                                          static_cast<__half*>(B));                              \
  } while (0)
  if (xtype == 0) VNM_CAST(__half);
  else if (xtype == 1) VNM_CAST(__nv_bfloat16);
  else VNM_CAST(float);
#undef VNM_CAST
  if (cudaGetLastError() != cudaSuccess) return VNM_ERR_CUDA;
  const vnm_status s = vnm_spmm_run_async(ctx, A, B, n, C, stream);
  ctx->launches++;
  return s;
}

vnm_status vnm_spmm_check(vnm_spmm_matrix* A, void* stream, int* failed) {
  if (!A || !failed) return VNM_ERR_ARG;
  *failed = 0;
  VNM_CUDA_TRY(cudaSetDevice(A->device));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int h = 0;
  VNM_CUDA_TRY(cudaMemcpyAsync(&h, A->err, sizeof(int), cudaMemcpyDeviceToHost, s));
  VNM_CUDA_TRY(cudaStreamSynchronize(s));
  VNM_CUDA_TRY(cudaMemsetAsync(A->err, 0, sizeof(int), s));
  *failed = h != 0;
  return VNM_OK;
}

}  // extern "C"
