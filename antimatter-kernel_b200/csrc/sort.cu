// Stable sort of (uint64 key, uint32 value) pairs.
//
// Small sets (kRankMax): every key's rank by comparison with all keys, two
// launches. Larger ones: LSD radix, 8 bits per pass, two launches per pass: a
// histogram of each tile's digits, and a scatter whose blocks add up the
// histograms before theirs (rows of tiles inside a group of 16, sums of whole
// groups), rank their tile's elements by warp match masks and stage it in
// digit order in shared memory, so that a digit's writes are contiguous. Each
// pass reads 20 B and writes 12 B per element; up to a million keys all of it
// stays in L2 and the launches and the dependent loads of a tile are what it
// takes, so tiles shrink with n until they fill the chip. Past kMaxTiles tiles
// (and in the allocation-free sort) the digit counters are scanned by kernels
// of their own.
#include <algorithm>

#include "amk_internal.cuh"

namespace amk {
namespace {

constexpr int kSortThreads = 256;
constexpr int kItems = 16;
constexpr int kTile = kSortThreads * kItems;
constexpr int kWarps = kSortThreads / 32;
// counters the one-CTA scan_kernel handles (64 per thread; the bound of the
// allocation-free sort, which has no scratch for the multi-CTA scan)
constexpr long kSingleScanCounters = 65536;

__global__ void __launch_bounds__(kSortThreads)
hist_kernel(const uint64_t* __restrict__ keys, long n, int shift, int nb, uint32_t* __restrict__ hist) {
  __shared__ uint32_t h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  const long base = static_cast<long>(blockIdx.x) * kTile;
#pragma unroll 4
  for (int k = 0; k < kItems; ++k) {
    const long i = base + k * kSortThreads + threadIdx.x;
    if (i < n) atomicAdd(&h[(keys[i] >> shift) & 0xFF], 1u);
  }
  __syncthreads();
  hist[static_cast<long>(threadIdx.x) * nb + blockIdx.x] = h[threadIdx.x];
}

// Exclusive scan of `len` counters with one CTA of 1024 threads.
__global__ void __launch_bounds__(1024) scan_kernel(uint32_t* __restrict__ data, long len) {
  __shared__ uint32_t s[1024];
  const long per = (len + 1023) / 1024;
  const long b = threadIdx.x * per;
  const long e = min(len, b + per);
  uint32_t sum = 0;
  for (long i = b; i < e; ++i) sum += data[i];
  s[threadIdx.x] = sum;
  __syncthreads();
  for (int off = 1; off < 1024; off <<= 1) {
    uint32_t v = threadIdx.x >= off ? s[threadIdx.x - off] : 0u;
    __syncthreads();
    s[threadIdx.x] += v;
    __syncthreads();
  }
  uint32_t run = s[threadIdx.x] - sum;
  for (long i = b; i < e; ++i) {
    const uint32_t v = data[i];
    data[i] = run;
    run += v;
  }
}

__global__ void __launch_bounds__(kSortThreads)
scatter_kernel(const uint64_t* __restrict__ kin, const uint32_t* __restrict__ vin, long n, int shift, int nb,
               const uint32_t* __restrict__ offs, uint64_t* __restrict__ kout, uint32_t* __restrict__ vout) {
  __shared__ uint32_t cnt[kWarps][256];
  __shared__ uint32_t running[256];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  running[threadIdx.x] = 0;
  const uint32_t base_off = 0;
  (void)base_off;
  const long base = static_cast<long>(blockIdx.x) * kTile;
  const uint32_t lt_mask = (1u << lane) - 1u;
  for (int k = 0; k < kItems; ++k) {
    const long i = base + k * kSortThreads + threadIdx.x;
    const bool valid = i < n;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) cnt[w][threadIdx.x] = 0;
    __syncthreads();
    uint64_t key = 0;
    uint32_t val = 0;
    int d = 0;
    uint32_t rank = 0;
    const uint32_t active = __ballot_sync(0xffffffffu, valid);
    if (valid) {
      key = kin[i];
      val = vin[i];
      d = static_cast<int>((key >> shift) & 0xFF);
      const uint32_t peers = __match_any_sync(active, d);
      rank = __popc(peers & lt_mask);
      if ((peers & lt_mask) == 0) cnt[warp][d] = __popc(peers);
    }
    __syncthreads();
    if (valid) {
      uint32_t pre = running[d] + rank;
      for (int w = 0; w < warp; ++w) pre += cnt[w][d];
      const long pos = static_cast<long>(offs[static_cast<long>(d) * nb + blockIdx.x]) + pre;
      kout[pos] = key;
      vout[pos] = val;
    }
    __syncthreads();
    uint32_t add = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) add += cnt[w][threadIdx.x];
    running[threadIdx.x] += add;
    __syncthreads();
  }
}

// ---------------------------------------------------------------- radix, two launches per pass
constexpr int kGroup = 16;         // tiles per group of the second level
constexpr long kMaxTiles = 4096;   // 256 groups of 1 KB to add per block at most

template <int kI>
__global__ void __launch_bounds__(kSortThreads)
tile_hist_kernel(const uint64_t* __restrict__ keys, long n, int shift, uint32_t* __restrict__ rows,
                 uint32_t* __restrict__ groups) {
  __shared__ uint32_t h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  const long base = static_cast<long>(blockIdx.x) * (kSortThreads * kI);
#pragma unroll
  for (int k = 0; k < kI; ++k) {
    const long i = base + k * kSortThreads + threadIdx.x;
    if (i < n) atomicAdd(&h[(keys[i] >> shift) & 0xFF], 1u);
  }
  __syncthreads();
  const uint32_t c = h[threadIdx.x];
  rows[static_cast<size_t>(blockIdx.x) * 256 + threadIdx.x] = c;
  if (c) atomicAdd(&groups[static_cast<size_t>(blockIdx.x / kGroup) * 256 + threadIdx.x], c);
}

// Sum over the block's warps before this one of a per-thread value's warp
// total, plus the exclusive scan inside the warp: exclusive block scan.
__device__ __forceinline__ uint32_t block_exclusive(uint32_t v, uint32_t* wsum) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  __syncthreads();  // wsum is free
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  uint32_t before = 0;
  for (int w = 0; w < warp; ++w) before += wsum[w];
  return before + incl - v;
}

template <int kI>
constexpr size_t staged_smem() {
  return static_cast<size_t>(kSortThreads) * kI * (sizeof(uint64_t) + sizeof(uint32_t)) +
         sizeof(uint32_t) * (kWarps * 256 + 256 + kWarps);
}

// offs (digit-major, scanned) gives digit d of this tile its first place, or
// (offs null) the rows and groups of tile_hist_kernel do. Warp w ranks the
// contiguous chunk w of the tile with counters of its own (match masks per
// round, no block barrier), which keeps the ranks stable; one block pass then
// turns the per-warp digit counts into tile positions, the elements are placed
// in shared memory in sorted order and written out in that order. Element j of
// the staged tile goes to first[d] + j - (tile start of digit d).
template <int kI>
__global__ void __launch_bounds__(kSortThreads)
scatter_staged_kernel(const uint64_t* __restrict__ kin, const uint32_t* __restrict__ vin, long n, int shift,
                      int nb, const uint32_t* __restrict__ offs, const uint32_t* __restrict__ rows,
                      const uint32_t* __restrict__ groups, uint64_t* __restrict__ kout,
                      uint32_t* __restrict__ vout) {
  constexpr int kT = kSortThreads * kI, kChunk = kT / kWarps;
  extern __shared__ __align__(16) unsigned char sort_smem[];
  uint64_t* sk = reinterpret_cast<uint64_t*>(sort_smem);
  uint32_t* sv = reinterpret_cast<uint32_t*>(sk + kT);
  uint32_t* wc = sv + kT;                    // [kWarps][256]: counts, then tile positions
  uint32_t* first = wc + kWarps * 256;       // [256]: place of digit d minus its tile start
  uint32_t* wsum = first + 256;              // [kWarps]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long base = static_cast<long>(blockIdx.x) * kT;
  const long wbase = base + static_cast<long>(warp) * kChunk;
  const uint32_t lt_mask = (1u << lane) - 1u;
  uint32_t* mine = wc + warp * 256;
  uint64_t key[kI];
  uint32_t val[kI], dr[kI];  // dr: digit | rank in the warp's chunk << 8
#pragma unroll
  for (int k = 0; k < kI; ++k) {
    const long i = wbase + k * 32 + lane;
    key[k] = i < n ? kin[i] : 0;
    val[k] = i < n ? vin[i] : 0;
  }
  for (int d = lane; d < 256; d += 32) mine[d] = 0;
  // digit d = thread d: its place in the output before this tile
  uint32_t place;
  if (offs) {
    place = offs[static_cast<size_t>(threadIdx.x) * nb + blockIdx.x];
  } else {
    const int my = blockIdx.x / kGroup, n_groups = (nb + kGroup - 1) / kGroup;
    uint32_t before = 0, total = 0;
#pragma unroll 8
    for (int g = 0; g < n_groups; ++g) {
      const uint32_t c = groups[static_cast<size_t>(g) * 256 + threadIdx.x];
      total += c;
      if (g < my) before += c;
    }
#pragma unroll 8
    for (int r = my * kGroup; r < static_cast<int>(blockIdx.x); ++r)
      before += rows[static_cast<size_t>(r) * 256 + threadIdx.x];
    place = block_exclusive(total, wsum) + before;
  }
  __syncwarp();
#pragma unroll
  for (int k = 0; k < kI; ++k) {
    const bool valid = wbase + k * 32 + lane < n;
    dr[k] = 0;
    const uint32_t active = __ballot_sync(0xffffffffu, valid);
    if (valid) {
      const int d = static_cast<int>((key[k] >> shift) & 0xFF);
      const uint32_t peers = __match_any_sync(active, d);
      const int leader = __ffs(peers) - 1;
      uint32_t old = lane == leader ? mine[d] : 0u;
      old = __shfl_sync(active, old, leader);
      if (lane == leader) mine[d] = old + __popc(peers);
      dr[k] = static_cast<uint32_t>(d) | ((old + __popc(peers & lt_mask)) << 8);
    }
    __syncwarp();
  }
  __syncthreads();
  // digit d (thread d): the per-warp starts within the digit and the digit's total
  {
    const int d = threadIdx.x;
    uint32_t run = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const uint32_t c = wc[w * 256 + d];
      wc[w * 256 + d] = run;
      run += c;
    }
    const uint32_t start = block_exclusive(run, wsum);
    first[d] = place - start;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) wc[w * 256 + d] += start;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kI; ++k) {
    if (wbase + k * 32 + lane < n) {
      const uint32_t pos = mine[dr[k] & 0xFF] + (dr[k] >> 8);
      sk[pos] = key[k];
      sv[pos] = val[k];
    }
  }
  __syncthreads();
  const int tile_n = static_cast<int>(min(static_cast<long>(kT), n - base));
#pragma unroll 4
  for (int j = threadIdx.x; j < tile_n; j += kSortThreads) {
    const uint64_t kk = sk[j];
    const uint32_t pos = first[(kk >> shift) & 0xFF] + static_cast<uint32_t>(j);
    kout[pos] = kk;
    vout[pos] = sv[j];
  }
}

// ---------------------------------------------------------------- ranks
// Up to this many keys the comparisons are cheaper than the passes: us per
// 63-bit sort, ranks / 8 passes: 500 keys 19 / 93, 5,000 29 / 88, 12,000
// 51 / 100, 16,384 73 / 104, 20,000 98 / 102, 32,768 205 / 102. (With five
// launches per pass 210 us at 30,000 and 288 us at 524,309 keys, where the
// two-launch passes take 103 and 165.)
constexpr long kRankMax = 16384;
constexpr int kRankSeg = 1024;  // keys a block compares its 256 elements with

// rank[i] += keys of segment blockIdx.y before key i (ties by index)
__global__ void __launch_bounds__(kSortThreads)
rank_kernel(const uint64_t* __restrict__ keys, int n, uint64_t mask, int* __restrict__ rank) {
  __shared__ uint64_t s[kRankSeg];
  const int j0 = blockIdx.y * kRankSeg, cnt = min(kRankSeg, n - j0);
  for (int j = threadIdx.x; j < cnt; j += kSortThreads) s[j] = keys[j0 + j] & mask;
  __syncthreads();
  const int i = blockIdx.x * kSortThreads + threadIdx.x;
  if (i >= n) return;
  const uint64_t k = keys[i] & mask;
  int r = 0;
  if (j0 + cnt <= static_cast<int>(blockIdx.x) * kSortThreads) {  // all before: ties count
#pragma unroll 8
    for (int j = 0; j < cnt; ++j) r += s[j] <= k ? 1 : 0;
  } else if (j0 > i) {  // all after
#pragma unroll 8
    for (int j = 0; j < cnt; ++j) r += s[j] < k ? 1 : 0;
  } else {
#pragma unroll 8
    for (int j = 0; j < cnt; ++j) r += s[j] < k || (s[j] == k && j0 + j < i) ? 1 : 0;
  }
  if (r) atomicAdd(rank + i, r);
}

__global__ void rank_scatter_kernel(const uint64_t* __restrict__ kin, const uint32_t* __restrict__ vin, int n,
                                    const int* __restrict__ rank, uint64_t* __restrict__ kout,
                                    uint32_t* __restrict__ vout) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  kout[rank[i]] = kin[i];
  vout[rank[i]] = vin[i];
}

}  // namespace

namespace {

template <int kI>
int radix_passes(amk_ctx* c, const uint64_t* ksrc, const uint32_t* vsrc, uint64_t* keys_out, uint32_t* vals_out,
                 uint64_t* kt, uint32_t* vt, long n, int passes) {
  const int nb = static_cast<int>((n + kSortThreads * kI - 1) / (kSortThreads * kI));
  const bool own = nb <= kMaxTiles;
  const size_t n_groups = static_cast<size_t>((nb + kGroup - 1) / kGroup);
  int rc = AMK_OK;
  // rows (or digit-major counters), then the groups of every pass
  uint32_t* rows = slot<uint32_t>(c, kSlotSortHist, 256 * (static_cast<size_t>(nb) + (own ? passes * n_groups : 0)), &rc);
  AMK_TRY(rc);
  uint32_t* groups = rows + 256 * static_cast<size_t>(nb);
  int* total = slot<int>(c, kSlotSortFlags, 8, &rc);
  AMK_TRY(rc);
  // the staged scatter's shared memory may be above the 48 KB default (set per call: per device)
  AMK_CUDA_TRY(cudaFuncSetAttribute(scatter_staged_kernel<kI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    static_cast<int>(staged_smem<kI>())));
  if (own) AMK_CUDA_TRY(cudaMemsetAsync(groups, 0, 256 * sizeof(uint32_t) * passes * n_groups, c->stream));
  for (int p = 0; p < passes; ++p) {
    const bool to_out = ((passes - 1 - p) % 2) == 0;
    uint64_t* kdst = to_out ? keys_out : kt;
    uint32_t* vdst = to_out ? vals_out : vt;
    const int shift = 8 * p;
    uint32_t* gp = groups + 256 * n_groups * p;
    if (own) {
      tile_hist_kernel<kI><<<nb, kSortThreads, 0, c->stream>>>(ksrc, n, shift, rows, gp);
      AMK_TRY(check_launch(c, "tile_hist_kernel"));
    } else {
      hist_kernel<<<nb, kSortThreads, 0, c->stream>>>(ksrc, n, shift, nb, rows);  // kItems = the largest kI
      AMK_TRY(check_launch(c, "hist_kernel"));
      // in place; counts stay below 2^31
      AMK_TRY(exclusive_scan_int(c, reinterpret_cast<const int*>(rows), static_cast<long>(256) * nb,
                                 reinterpret_cast<int*>(rows), total));
    }
    scatter_staged_kernel<kI><<<nb, kSortThreads, staged_smem<kI>(), c->stream>>>(
        ksrc, vsrc, n, shift, nb, own ? nullptr : rows, rows, gp, kdst, vdst);
    AMK_TRY(check_launch(c, "scatter_staged_kernel"));
    ksrc = kdst;
    vsrc = vdst;
  }
  return AMK_OK;
}

}  // namespace

// Tiles of 1,024 keys up to 150,000 (147 of them: one per SM), 2,048 up to
// 600,000, 4,096 above.
int radix_sort_pairs(amk_ctx* c, const uint64_t* keys_in, const uint32_t* vals_in, uint64_t* keys_out,
                     uint32_t* vals_out, long n, int key_bits) {
  if (n <= 0) return AMK_OK;
  if (n > 0xFFFFFFF0L) return fail(AMK_ERR_LIMIT, "radix sort of %ld elements exceeds 32-bit ranks", n);
  const int passes = std::max(1, (key_bits + 7) / 8);
  int rc = AMK_OK;
  if (n <= kRankMax) {
    int* rank = slot<int>(c, kSlotValsB, static_cast<size_t>(n), &rc);
    AMK_TRY(rc);
    const uint64_t mask = passes >= 8 ? ~0ull : (1ull << (8 * passes)) - 1ull;
    const unsigned gb = static_cast<unsigned>((n + kSortThreads - 1) / kSortThreads);
    AMK_CUDA_TRY(cudaMemsetAsync(rank, 0, static_cast<size_t>(n) * sizeof(int), c->stream));
    rank_kernel<<<dim3(gb, static_cast<unsigned>((n + kRankSeg - 1) / kRankSeg)), kSortThreads, 0, c->stream>>>(
        keys_in, static_cast<int>(n), mask, rank);
    AMK_TRY(check_launch(c, "rank_kernel"));
    rank_scatter_kernel<<<gb, kSortThreads, 0, c->stream>>>(keys_in, vals_in, static_cast<int>(n), rank, keys_out,
                                                            vals_out);
    return check_launch(c, "rank_scatter_kernel");
  }
  uint64_t* kt = slot<uint64_t>(c, kSlotKeysB, static_cast<size_t>(n), &rc);
  AMK_TRY(rc);
  uint32_t* vt = slot<uint32_t>(c, kSlotValsB, static_cast<size_t>(n), &rc);
  AMK_TRY(rc);
  if (n <= 150000) return radix_passes<4>(c, keys_in, vals_in, keys_out, vals_out, kt, vt, n, passes);
  if (n <= 600000) return radix_passes<8>(c, keys_in, vals_in, keys_out, vals_out, kt, vt, n, passes);
  return radix_passes<16>(c, keys_in, vals_in, keys_out, vals_out, kt, vt, n, passes);
}

}  // namespace amk

namespace amk {

// The same sort on caller-provided buffers (no context, no allocation):
// ktmp/vtmp hold n elements, hist holds 256 * ceil(n / 4096) counters. The
// digit scan is the one-CTA scan_kernel, so 256 * ceil(n / 4096) must stay
// within kSingleScanCounters (n <= 1,048,576): larger n is refused with
// cudaErrorInvalidValue before anything is launched.
cudaError_t radix_sort_pairs_buffers(cudaStream_t stream, const uint64_t* keys_in, const uint32_t* vals_in,
                                     uint64_t* keys_out, uint32_t* vals_out, uint64_t* ktmp, uint32_t* vtmp,
                                     uint32_t* hist, long n, int key_bits) {
  if (n <= 0) return cudaSuccess;
  const int passes = std::max(1, (key_bits + 7) / 8);
  const int nb = static_cast<int>((n + kTile - 1) / kTile);
  if (static_cast<long>(256) * nb > kSingleScanCounters) return cudaErrorInvalidValue;
  const uint64_t* ksrc = keys_in;
  const uint32_t* vsrc = vals_in;
  for (int p = 0; p < passes; ++p) {
    const bool to_out = ((passes - 1 - p) % 2) == 0;
    uint64_t* kdst = to_out ? keys_out : ktmp;
    uint32_t* vdst = to_out ? vals_out : vtmp;
    const int shift = 8 * p;
    hist_kernel<<<nb, kSortThreads, 0, stream>>>(ksrc, n, shift, nb, hist);
    scan_kernel<<<1, 1024, 0, stream>>>(hist, static_cast<long>(256) * nb);
    scatter_kernel<<<nb, kSortThreads, 0, stream>>>(ksrc, vsrc, n, shift, nb, hist, kdst, vdst);
    ksrc = kdst;
    vsrc = vdst;
  }
  return cudaGetLastError();
}

}  // namespace amk
