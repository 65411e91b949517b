// Device-wide exclusive scan and stable LSD radix sort of (64-bit key, 32-bit value) pairs.
//
// Used by the Gaussian rasteriser to order the (tile, depth) keys of views with very full tiles (the reference's rasteriser extension,
// opt_gaussian_rasterization, uses CUB for this; call site benchmarks/nerf/origin_gs/gs_model.py:211-220)
// and by the atomic-free grid backward.  All temporary storage is provided by the caller as one
// scratch buffer, so a call performs no allocation.
//
// Sort pass (8-bit digit): a block ranks the keys of its tile (equal digits of a warp by __match_any_sync, warps through
// shared-memory counters - stable by construction), orders the tile in shared memory and writes runs of equal digits.  Where
// a digit's run goes depends on the tiles before: small inputs learn it from the counts those publish (decoupled look-back;
// one kernel counts the digits of every pass beforehand, then a pass is one kernel), large ones from a count per tile and a
// scan over [256][tiles], because the look-back of many tiles reads their counts over and over.
#include "common.cuh"
#include <algorithm>

namespace lmb {

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kDigits = 256;
constexpr int kMaxPasses = 8;
constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

// ---- scan -------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* smem, uint32_t& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
    if (lane >= d) x += y;
  }
  if (lane == 31) smem[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = lane < (blockDim.x >> 5) ? smem[lane] : 0;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, w, d);
      if (lane >= d) w += y;
    }
    smem[lane] = w;
  }
  __syncthreads();
  const uint32_t warp_base = warp ? smem[warp - 1] : 0;
  total = smem[(blockDim.x >> 5) - 1];
  __syncthreads();
  return warp_base + x - v;
}

__global__ void __launch_bounds__(kScanThreads)
scan_tiles_kernel(const uint32_t* in, uint32_t* out, uint32_t* __restrict__ tile_sums, long long n) {
  // `out` may be the same buffer as `in` (the recursion scans the tile sums in place): a thread loads all of its
  // items before it stores any, and it stores only to the positions it loaded, so the two are not marked restrict.
  __shared__ uint32_t sm[32];
  const long long base = (long long)blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  uint32_t v[kScanItems], sum = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) { v[i] = (base + i < n) ? in[base + i] : 0; sum += v[i]; }
  uint32_t total;
  uint32_t excl = block_excl_scan(sum, sm, total);
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) { if (base + i < n) out[base + i] = excl; excl += v[i]; }
  if (threadIdx.x == 0 && tile_sums) tile_sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanThreads)
scan_add_kernel(uint32_t* __restrict__ out, const uint32_t* __restrict__ tile_offsets, long long n) {
  const uint32_t off = tile_offsets[blockIdx.x];
  const long long base = (long long)blockIdx.x * kScanTile + threadIdx.x * kScanItems;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) if (base + i < n) out[base + i] += off;
}

// scratch layout for scan of n items: level-1 sums (ceil(n/T)), level-2 sums (ceil(l1/T)), ...
static long long scan_scratch_elems(long long n) {
  long long total = 0;
  while (n > kScanTile) { n = (n + kScanTile - 1) / kScanTile; total += n; }
  return total + 1;
}

static int exclusive_scan(const uint32_t* in, uint32_t* out, long long n, uint32_t* scratch, cudaStream_t stream) {
  const long long tiles = (n + kScanTile - 1) / kScanTile;
  if (tiles <= 1) {
    scan_tiles_kernel<<<1, kScanThreads, 0, stream>>>(in, out, nullptr, n);
    LMB_LAUNCH_CHECK();
    return 0;
  }
  scan_tiles_kernel<<<(int)tiles, kScanThreads, 0, stream>>>(in, out, scratch, n);
  LMB_LAUNCH_CHECK();
  int rc = exclusive_scan(scratch, scratch, tiles, scratch + tiles, stream);
  if (rc) return rc;
  scan_add_kernel<<<(int)tiles, kScanThreads, 0, stream>>>(out, scratch, n);
  LMB_LAUNCH_CHECK();
  return 0;
}

// ---- radix sort ----------------------------------------------------------------------------------------
static_assert(kSortThreads == kDigits, "one thread per digit");

// hist[pass][digit] += keys of this block's share; one read of the keys for all passes
__global__ void __launch_bounds__(kSortThreads)
radix_hist_kernel(const uint64_t* __restrict__ keys, const int* __restrict__ count_ptr, long long max_n, int begin_bit, int passes,
                  uint32_t* __restrict__ hist) {
  __shared__ uint32_t h[kMaxPasses][kDigits];
  for (int p = 0; p < passes; ++p) h[p][threadIdx.x] = 0;
  __syncthreads();
  const long long n = resolve_count(count_ptr, max_n);
  const long long step = (long long)gridDim.x * kSortThreads;
  for (long long i = (long long)blockIdx.x * kSortThreads + threadIdx.x; i < n; i += step) {
    const uint64_t key = keys[i] >> begin_bit;
#pragma unroll
    for (int p = 0; p < kMaxPasses; ++p)
      if (p < passes) atomicAdd(&h[p][(key >> (8 * p)) & 0xFF], 1u);
  }
  __syncthreads();
  for (int p = 0; p < passes; ++p)
    if (h[p][threadIdx.x]) atomicAdd(&hist[p * kDigits + threadIdx.x], h[p][threadIdx.x]);
}

// counts[digit][tile] of one pass, totals[digit] += (zeroed before)
template <int kItems>
__global__ void __launch_bounds__(kSortThreads)
radix_count_kernel(const uint64_t* __restrict__ keys, const int* __restrict__ count_ptr, long long max_n, int shift,
                   uint32_t* __restrict__ counts, uint32_t* __restrict__ totals, int tiles) {
  __shared__ uint32_t h[kDigits];
  h[threadIdx.x] = 0;
  __syncthreads();
  const long long n = resolve_count(count_ptr, max_n), first = (long long)blockIdx.x * kSortThreads * kItems;
  uint64_t key[kItems];
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    const long long i = first + k * kSortThreads + threadIdx.x;
    key[k] = i < n ? keys[i] : 0;
  }
#pragma unroll
  for (int k = 0; k < kItems; ++k)
    if (first + k * kSortThreads + threadIdx.x < n) atomicAdd(&h[(key[k] >> shift) & 0xFF], 1u);
  __syncthreads();
  counts[(long long)threadIdx.x * tiles + blockIdx.x] = h[threadIdx.x];
  if (h[threadIdx.x]) atomicAdd(&totals[threadIdx.x], h[threadIdx.x]);
}

// counts[digit][tile] -> where the tile's keys of the digit start: one block per digit
__global__ void __launch_bounds__(kDigits)
radix_offsets_kernel(uint32_t* __restrict__ counts, const uint32_t* __restrict__ totals, int tiles) {
  __shared__ uint32_t sm[32];
  const int tid = threadIdx.x, digit = blockIdx.x;
  uint32_t carry, sum;
  block_excl_scan(tid < digit ? totals[tid] : 0u, sm, carry);
  uint32_t* row = counts + (long long)digit * tiles;
  for (int t0 = 0; t0 < tiles; t0 += 4 * kDigits) {
    uint32_t v[4], mine = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int t = t0 + 4 * tid + k;
      v[k] = t < tiles ? row[t] : 0u;
      mine += v[k];
    }
    uint32_t at = carry + block_excl_scan(mine, sm, sum);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int t = t0 + 4 * tid + k;
      if (t < tiles) row[t] = at;
      at += v[k];
    }
    carry += sum;
  }
}

// State of (tile, digit) in a pass: the low 30 bits hold a count, the two high bits say of what (0: not yet published, 1: the
// tile's own keys, 2: those of the tile and all before it).  One word carries both, so no fence is needed.
__device__ __forceinline__ void state_store(uint32_t* p, uint32_t kind, uint32_t count) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(kind << 30 | count) : "memory");
}
__device__ __forceinline__ uint32_t state_load(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

constexpr int kLookback = 16;         // predecessors fetched at once: a step of the walk costs one L2 round trip
constexpr int kSpinLimit = 1 << 16;   // polls of a walk; then the block counts the keys before it by itself

// Keys with digit `digit` before tile `tile`, from the published states; false when the walk gave up.
__device__ __forceinline__ bool look_back(const uint32_t* __restrict__ state, int tile, int digit, int spin_limit, uint32_t& before) {
  uint32_t sum = 0;
  int spins = 0;
  for (int t = tile - 1; t >= 0;) {
    uint32_t w[kLookback];
#pragma unroll
    for (int k = 0; k < kLookback; ++k) w[k] = state_load(state + (long long)max(t - k, 0) * kDigits + digit);
    int taken = 0;
    bool done = false;
#pragma unroll
    for (int k = 0; k < kLookback; ++k)
      if (!done && taken == k && t >= k && w[k] >> 30 != 0) {          // an unpublished state ends the step: the rest is polled again
        sum += w[k] & 0x3FFFFFFFu;
        taken = k + 1;
        done = w[k] >> 30 == 2;
      }
    if (done) break;
    t -= taken;
    if (taken == 0 && ++spins > spin_limit) return false;
  }
  before = sum;
  return true;
}

// Lanes that hold the same digit, from one ballot per bit.  (__match_any_sync takes its time per distinct value: with 30
// different digits in a warp it was three quarters of a pass.)
__device__ __forceinline__ uint32_t same_digit(uint32_t digit, bool valid) {
  uint32_t peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const uint32_t ones = __ballot_sync(0xffffffffu, digit >> b & 1u);
    peers &= digit >> b & 1u ? ones : ~ones;
  }
  return peers;
}

template <int kItems>
struct SortTile {
  uint64_t keys[kSortThreads * kItems];
  uint32_t vals[kSortThreads * kItems];
  uint32_t cnt[kSortWarps][kDigits];    // keys of a digit per warp, then where a warp's first of them goes in the tile
  uint32_t base[kDigits];               // global position of the tile's first key of a digit, minus its position in the tile
  uint32_t scan[32];
  int tile, redo;                       // look-back only
};

// One pass.  kScanned: offsets[digit][tile] holds where the tile's first key of a digit goes; otherwise hist holds the digits'
// counts of the whole input, and ticket and state serve the look-back.  Bound by memory (24 B per pair) for large inputs and by
// the walk and launches for small ones.  Whole sort on 45 bits, random keys: 20 k pairs 174 -> 72 us, 150 k 224 -> 85, 1 M
// 246 -> 130, 4 M 541 -> 359, 12 M 1849 -> 956.  8 keys a thread keep four blocks on an SM where 16 keep three; with five the
// compiler spills (a pass of a frame of 6 M Gaussians 46.0 against 45.0 us, of 0.4 M anchors 16.7 against 15.8).
template <int kItems, bool kScanned>
__global__ void __launch_bounds__(kSortThreads, kItems > 8 ? 3 : 4)
radix_pass_kernel(const uint64_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in, uint64_t* __restrict__ keys_out,
                  uint32_t* __restrict__ vals_out, const int* __restrict__ count_ptr, long long max_n, int shift,
                  const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ hist, uint32_t* __restrict__ ticket,
                  uint32_t* __restrict__ state, int spin_limit) {
  constexpr int kTile = kSortThreads * kItems;
  extern __shared__ __align__(16) unsigned char smem[];
  SortTile<kItems>& s = *reinterpret_cast<SortTile<kItems>*>(smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (!kScanned && tid == 0) { s.tile = (int)atomicAdd(ticket, 1u); s.redo = 0; }
#pragma unroll
  for (int w = 0; w < kSortWarps; ++w) s.cnt[w][tid] = 0;
  __syncthreads();
  const int tile = kScanned ? (int)blockIdx.x : s.tile;      // tiles start in ticket order: every one before this is running
  const long long n = resolve_count(count_ptr, max_n);
  const long long first = (long long)tile * kTile;
  if (first >= n) return;
  const int count = (int)(n - first < kTile ? n - first : kTile);
  const int at = warp * 32 * kItems + lane;
  uint32_t* my_state = kScanned ? nullptr : state + (long long)tile * kDigits + tid;
  const uint32_t base = kScanned ? offsets[(long long)tid * gridDim.x + tile] : hist[tid];
  uint32_t own = 0, local;
  {
    // rank: a warp owns 32 * kItems consecutive keys, item k of its lanes is the k-th run of 32
    uint64_t key[kItems];
    uint32_t rank[kItems];
#pragma unroll
    for (int k = 0; k < kItems; ++k) key[k] = at + 32 * k < count ? keys_in[first + at + 32 * k] : 0;
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const bool valid = at + 32 * k < count;
      const uint32_t digit = (uint32_t)(key[k] >> shift) & 0xFF;
      const uint32_t peers = same_digit(digit, valid);
      const uint32_t lower = __popc(peers & ((1u << lane) - 1u));
      const uint32_t seen = valid ? s.cnt[warp][digit] : 0u;
      __syncwarp();
      if (valid && lower == 0) s.cnt[warp][digit] = seen + __popc(peers);
      __syncwarp();
      rank[k] = seen + lower;
    }
    __syncthreads();

    // thread d: count of digit d in the tile, published; its exclusive sum over digits places the digit inside the tile
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) { const uint32_t c = s.cnt[w][tid]; s.cnt[w][tid] = own; own += c; }
    if (!kScanned && tile > 0) state_store(my_state, 1, own);
    uint32_t total;
    local = block_excl_scan(own, s.scan, total);
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) s.cnt[w][tid] += local;
    __syncthreads();

    // order the tile in shared memory while the tiles before it publish theirs
#pragma unroll
    for (int k = 0; k < kItems; ++k)
      if (at + 32 * k < count) {
        const uint32_t pos = s.cnt[warp][(key[k] >> shift) & 0xFF] + rank[k];
        s.keys[pos] = key[k];
        s.vals[pos] = vals_in[first + at + 32 * k];
      }
  }
  if constexpr (kScanned) {
    s.base[tid] = base - local;
  } else {
    uint32_t total, before = 0;
    const uint32_t global = block_excl_scan(base, s.scan, total);
    if (!look_back(state, tile, tid, spin_limit, before)) s.redo = 1;
    __syncthreads();
    if (s.redo) {                                     // bounded wait ran out: count digits before the tile from the keys
      s.base[tid] = 0;
      __syncthreads();
      for (long long i = tid; i < first; i += kSortThreads) atomicAdd(&s.base[(keys_in[i] >> shift) & 0xFF], 1u);
      __syncthreads();
      before = s.base[tid];
      __syncthreads();
    }
    state_store(my_state, 2, before + own);
    s.base[tid] = global + before - local;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    const int i = tid + k * kSortThreads;
    if (i < count) {
      const uint64_t v = s.keys[i];
      const uint32_t pos = s.base[(v >> shift) & 0xFF] + i;
      keys_out[pos] = v;
      vals_out[pos] = s.vals[i];
    }
  }
}

}  // namespace lmb

using namespace lmb;

LMB_API long long lmb_scan_scratch_bytes(long long n) { return scan_scratch_elems(n) * 4; }

LMB_API int lmb_exclusive_scan_u32(const uint32_t* in, uint32_t* out, long long n, void* scratch, cudaStream_t stream) {
  if (n <= 0) return 0;
  return exclusive_scan(in, out, n, (uint32_t*)scratch, stream);
}

// Tiles of 4 keys a thread with the look-back while they are few, tiles of 16 with the look-back next (a third of the launches
// of the counted form), tiles of 8 with counted and scanned offsets from kCounted pairs on: the look-back of a wave of tiles
// reads their counts in proportion to the square of its size.  Whole sorts on 45 bits: 150 k pairs 85 us in tiles of 4 keys,
// 109 in tiles of 16, and the two meet at kFewPairs (96 us on either side).  At kCounted random keys still sort a little faster
// with the look-back (151 against 174 us), but the runs of equal digits of a frame's keys do not: a training step's sort (a
// capacity of 1.5 to 3 M pairs) took 456 us with it and takes 155 counted.  Counted in tiles of 16: 2 M pairs 230 us, 4 M 396,
// 12 M 1066; in tiles of 8: 196, 359, 956.
constexpr long long kFewPairs = 1LL << 18, kCounted = 5LL << 18;

struct SortPlan {
  int items;
  bool counted;
  long long tiles, vals_alt, counts, state, bytes;     // offsets; the alternate keys come first
  explicit SortPlan(long long max_n) {
    counted = max_n >= kCounted;
    items = max_n < kFewPairs ? 4 : counted ? 8 : 16;
    tiles = (max_n + kSortThreads * items - 1) / (kSortThreads * items);
    vals_alt = max_n * 8;
    counts = (max_n * 12 + 255) & ~255LL;              // digit counts of all passes, tickets
    state = counts + kMaxPasses * kDigits * 4 + 256;   // states of all passes' tiles, or one pass's counts
    bytes = state + (counted ? 1 : kMaxPasses) * tiles * kDigits * 4;
  }
};

// Bytes of scratch needed to sort up to max_n pairs: the alternate key/value buffers, the digits' counts and those of the tiles.
LMB_API long long lmb_radix_sort_scratch_bytes(long long max_n) {
  long long bytes = SortPlan(max_n).bytes;              // and enough for any shorter input
  if (max_n >= kFewPairs) bytes = std::max(bytes, SortPlan(kFewPairs - 1).bytes);
  if (max_n >= kCounted) bytes = std::max(bytes, SortPlan(kCounted - 1).bytes);
  return bytes + 256;
}

template <int kItems, bool kScanned>
static int radix_pass(const uint64_t* kin, const uint32_t* vin, uint64_t* kout, uint32_t* vout, const int* count_ptr, long long max_n,
                      int shift, long long tiles, const uint32_t* offsets, const uint32_t* hist, uint32_t* ticket, uint32_t* state,
                      int spin_limit, cudaStream_t stream) {
  constexpr int smem = sizeof(SortTile<kItems>);
  LMB_CUDA_TRY(cudaFuncSetAttribute(radix_pass_kernel<kItems, kScanned>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  radix_pass_kernel<kItems, kScanned><<<(int)tiles, kSortThreads, smem, stream>>>(kin, vin, kout, vout, count_ptr, max_n, shift, offsets,
                                                                                 hist, ticket, state, spin_limit);
  LMB_LAUNCH_CHECK();
  return 0;
}

// As below; spin_limit bounds the polls of a block's walk over its predecessors (the result does not depend on it).
LMB_API int lmb_radix_sort_pairs_bounded(uint64_t* keys, uint32_t* vals, const int* count_ptr, long long max_n, int begin_bit,
                                         int end_bit, void* scratch, int spin_limit, cudaStream_t stream) {
  if (max_n <= 0 || end_bit <= begin_bit) return 0;
  const int passes = (end_bit - begin_bit + 7) / 8;
  if (passes > kMaxPasses) return (int)cudaErrorInvalidValue;
  const SortPlan plan(max_n);
  unsigned char* p = (unsigned char*)(((uintptr_t)scratch + 255) & ~(uintptr_t)255);
  uint64_t *kin = keys, *kout = (uint64_t*)p;
  uint32_t *vin = vals, *vout = (uint32_t*)(p + plan.vals_alt);
  uint32_t *hist = (uint32_t*)(p + plan.counts), *state = (uint32_t*)(p + plan.state);
  LMB_CUDA_TRY(cudaMemsetAsync(hist, 0, (plan.counted ? plan.state : plan.bytes) - plan.counts, stream));
  if (!plan.counted) {
    const long long want = (max_n + 16 * kSortThreads - 1) / (16 * kSortThreads);
    radix_hist_kernel<<<(int)want, kSortThreads, 0, stream>>>(kin, count_ptr, max_n, begin_bit, passes, hist);
    LMB_LAUNCH_CHECK();
  }
  for (int pass = 0; pass < passes; ++pass) {
    const int shift = begin_bit + 8 * pass;
    uint32_t* total = hist + pass * kDigits;
    int rc;
    if (plan.counted) {
      radix_count_kernel<8><<<(int)plan.tiles, kSortThreads, 0, stream>>>(kin, count_ptr, max_n, shift, state, total, (int)plan.tiles);
      LMB_LAUNCH_CHECK();
      radix_offsets_kernel<<<kDigits, kDigits, 0, stream>>>(state, total, (int)plan.tiles);
      LMB_LAUNCH_CHECK();
      rc = radix_pass<8, true>(kin, vin, kout, vout, count_ptr, max_n, shift, plan.tiles, state, nullptr, nullptr, nullptr, 0, stream);
    } else {
      const auto run = plan.items == 4 ? radix_pass<4, false> : radix_pass<16, false>;
      rc = run(kin, vin, kout, vout, count_ptr, max_n, shift, plan.tiles, nullptr, total, hist + kMaxPasses * kDigits + pass,
               state + pass * plan.tiles * kDigits, spin_limit, stream);
    }
    if (rc) return rc;
    uint64_t* tk = kin; kin = kout; kout = tk;
    uint32_t* tv = vin; vin = vout; vout = tv;
  }
  if (passes & 1) {
    LMB_CUDA_TRY(cudaMemcpyAsync(keys, kin, max_n * 8, cudaMemcpyDeviceToDevice, stream));
    LMB_CUDA_TRY(cudaMemcpyAsync(vals, vin, max_n * 4, cudaMemcpyDeviceToDevice, stream));
  }
  return 0;
}

// Sorts (keys, vals) in place (the result lands back in the input arrays) on bits [begin_bit, end_bit).
// (end_bit - begin_bit) is rounded up to a multiple of 8; an odd number of passes costs one copy back.
LMB_API int lmb_radix_sort_pairs(uint64_t* keys, uint32_t* vals, const int* count_ptr, long long max_n, int begin_bit,
                                 int end_bit, void* scratch, cudaStream_t stream) {
  return lmb_radix_sort_pairs_bounded(keys, vals, count_ptr, max_n, begin_bit, end_bit, scratch, kSpinLimit, stream);
}

// ---- allocation-free scan entry point (declared in lmb_noalloc.h) ---------------------------------------
#include <mutex>
#include "lmb_noalloc.h"

namespace {

// Workspace of the allocation-free scan.  It lives in every CUDA context that loads this library
// (LMB_NOALLOC_SCAN_SCRATCH_BYTES per GPU, until the process exits) and is shared by all calls.
static __device__ __align__(256) unsigned char g_noalloc_scan_scratch[LMB_NOALLOC_SCAN_SCRATCH_BYTES];

constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mutex;
void* g_noalloc_scratch_ptr[kMaxDevices] = {nullptr};

// Resolve the device address of the workspace for the current device.  The array's name is only a
// host-side handle in host code; the address a kernel can use has to come from the runtime.
int noalloc_scratch_for_current_device(void** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= kMaxDevices) return LMB_NOALLOC_ERR_DEVICE;
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (g_noalloc_scratch_ptr[dev] == nullptr) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scan_scratch);
    if (e != cudaSuccess) return (int)e;
    g_noalloc_scratch_ptr[dev] = p;
  }
  *out = g_noalloc_scratch_ptr[dev];
  return 0;
}

}  // namespace

LMB_API int lmb_exclusive_scan_u32_noalloc(const uint32_t* in, uint32_t* out, long long n, cudaStream_t stream) {
  if (n < 0 || in == nullptr || out == nullptr) return LMB_NOALLOC_ERR_ARGUMENT;
  if (n == 0) return 0;
  if (n > LMB_NOALLOC_SCAN_MAX_ELEMS || scan_scratch_elems(n) * 4 > (long long)LMB_NOALLOC_SCAN_SCRATCH_BYTES)
    return LMB_NOALLOC_ERR_TOO_LARGE;
  void* scratch = nullptr;
  const int rc = noalloc_scratch_for_current_device(&scratch);
  if (rc != 0) return rc;
  // Every workspace word that is read (per-tile sums of each level) is written earlier in the same
  // call, so nothing has to be cleared even though the array keeps the previous call's contents.
  return exclusive_scan(in, out, n, (uint32_t*)scratch, stream);
}
