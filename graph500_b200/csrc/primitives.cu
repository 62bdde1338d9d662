// Device primitives used by graph construction: error plumbing, allocation,
// an exclusive prefix sum (the reference's prefix_sum role,
// graph_constructor.hpp:404-408 and :486-491) and a stable LSD radix sort
// (the role of sort2 / std::sort in graph_constructor.hpp:318-322, :1376-1412).
#include "g500_internal.cuh"

#include <algorithm>
#include <mutex>

namespace g500 {

static thread_local std::string tl_error;

const char* last_error_text() { return tl_error.c_str(); }

int set_error(int code, const char* fmt, ...) {
  char buf[1024];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  tl_error = buf;
  return code;
}

int cuda_error(cudaError_t e, const char* what, const char* file, int line) {
  int code = (e == cudaErrorMemoryAllocation) ? G500_E_NOMEM : G500_E_DEVICE;
  cudaGetLastError();  // a refused call is reported here, not by the next launch's check as well
  return set_error(code, "%s failed: %s (%s:%d)", what, cudaGetErrorString(e), file, line);
}

int num_sms() {
  int dev = 0, n = 0;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
  return n;
}

int dev_alloc(void** p, size_t bytes, const char* what) {
  *p = nullptr;
  cudaError_t e = cudaMalloc(p, bytes);
  if (e != cudaSuccess) {
    *p = nullptr;
    cudaGetLastError();
    return set_error(e == cudaErrorMemoryAllocation ? G500_E_NOMEM : G500_E_DEVICE,
                     "cudaMalloc(%zu bytes) for %s failed: %s", bytes, what, cudaGetErrorString(e));
  }
  return G500_OK;
}

void dev_free(void* p) {
  if (p) cudaFree(p);
}

// Pinned host memory costs up to 3 ms while a process holds none of it, and a
// few tens of microseconds otherwise.  So one page per device, taken at the
// first call and kept until the process ends, holds the pieces of PINNED_PAGE /
// PINNED_SLOT handles; further ones get an allocation of their own.  With that
// cost in each handle a SCALE 22 construction to the first search and back took
// 2 ms longer; with none of it the first search into host memory on a new handle
// paid it (SCALE 16: 3.3 ms instead of 0.5).
namespace {
constexpr size_t PINNED_PAGE = 64 << 10;
constexpr int PINNED_SLOTS = (int)(PINNED_PAGE / PINNED_SLOT);
constexpr int PINNED_DEVICES = 64;
struct PinnedPage {
  std::mutex mu;
  char* base = nullptr;
  uint64_t used[PINNED_SLOTS / 64] = {};
};
PinnedPage pinned_pages[PINNED_DEVICES];
}  // namespace

int pinned_slot(int device, void** p, const char* what) {
  *p = nullptr;
  if (device >= 0 && device < PINNED_DEVICES) {
    PinnedPage& page = pinned_pages[device];
    std::lock_guard<std::mutex> lk(page.mu);
    if (page.base) {  // gone if the program has reset the device since
      cudaPointerAttributes a;
      if (cudaPointerGetAttributes(&a, page.base) != cudaSuccess || a.type != cudaMemoryTypeHost) {
        cudaGetLastError();
        page.base = nullptr;
      }
    }
    if (!page.base) {
      void* m = nullptr;
      G500_CUDA(cudaHostAlloc(&m, PINNED_PAGE, cudaHostAllocDefault));
      page.base = static_cast<char*>(m);
      for (auto& w : page.used) w = 0;
    }
    for (int i = 0; i < PINNED_SLOTS; ++i) {
      if ((page.used[i / 64] >> (i % 64)) & 1u) continue;
      page.used[i / 64] |= uint64_t(1) << (i % 64);
      *p = page.base + (size_t)i * PINNED_SLOT;
      return G500_OK;
    }
  }
  const cudaError_t e = cudaHostAlloc(p, PINNED_SLOT, cudaHostAllocDefault);
  return e == cudaSuccess ? G500_OK : cuda_error(e, what, __FILE__, __LINE__);
}

void pinned_slot_free(int device, void* p) {
  if (!p) return;
  if (device >= 0 && device < PINNED_DEVICES) {
    PinnedPage& page = pinned_pages[device];
    std::lock_guard<std::mutex> lk(page.mu);
    if (page.base && p >= page.base && p < page.base + PINNED_PAGE) {
      const size_t i = (size_t)(static_cast<char*>(p) - page.base) / PINNED_SLOT;
      page.used[i / 64] &= ~(uint64_t(1) << (i % 64));
      return;
    }
  }
  cudaFreeHost(p);
}

// ---------------------------------------------------------------------------
// exclusive scan
// ---------------------------------------------------------------------------
constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

template <typename T>
__device__ __forceinline__ uint64_t load_val(const T* in, int64_t i, int64_t n) {
  return i < n ? (uint64_t)in[i] : 0ull;
}

// Block-wide exclusive scan of one value per thread; returns the prefix and
// the block total.
__device__ __forceinline__ uint64_t block_exclusive_scan(uint64_t v, uint64_t* total, uint64_t* sh_warp) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint64_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint64_t y = __shfl_up_sync(FULL_MASK, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sh_warp[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint64_t w = lane < (SCAN_THREADS / 32) ? sh_warp[lane] : 0ull;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint64_t y = __shfl_up_sync(FULL_MASK, w, o);
      if (lane >= o) w += y;
    }
    if (lane < (SCAN_THREADS / 32)) sh_warp[lane] = w;  // inclusive warp totals
  }
  __syncthreads();
  uint64_t warp_prefix = warp ? sh_warp[warp - 1] : 0ull;
  *total = sh_warp[SCAN_THREADS / 32 - 1];
  return warp_prefix + x - v;
}

template <typename T>
__global__ void __launch_bounds__(SCAN_THREADS) scan_reduce_kernel(const T* in, int64_t n, uint64_t* partial) {
  __shared__ uint64_t sh_warp[SCAN_THREADS / 32];
  const int64_t base = (int64_t)blockIdx.x * SCAN_TILE;
  uint64_t s = 0;
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; ++k) s += load_val(in, base + k * SCAN_THREADS + threadIdx.x, n);
  uint64_t total;
  block_exclusive_scan(s, &total, sh_warp);
  if (threadIdx.x == 0) partial[blockIdx.x] = total;
}

template <typename T>
__global__ void __launch_bounds__(SCAN_THREADS) scan_tile_kernel(const T* in, uint64_t* out, int64_t n,
                                                                 const uint64_t* block_offsets) {
  __shared__ uint64_t tile[SCAN_TILE];
  __shared__ uint64_t sh_warp[SCAN_THREADS / 32];
  const int64_t base = (int64_t)blockIdx.x * SCAN_TILE;
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    int idx = k * SCAN_THREADS + threadIdx.x;
    tile[idx] = load_val(in, base + idx, n);
  }
  __syncthreads();
  uint64_t v[SCAN_ITEMS], s = 0;
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    v[k] = tile[threadIdx.x * SCAN_ITEMS + k];
    s += v[k];
  }
  uint64_t total;
  uint64_t run = block_exclusive_scan(s, &total, sh_warp) + (block_offsets ? block_offsets[blockIdx.x] : 0ull);
  __syncthreads();
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    tile[threadIdx.x * SCAN_ITEMS + k] = run;
    run += v[k];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    int64_t i = base + k * SCAN_THREADS + threadIdx.x;
    if (i < n) out[i] = tile[k * SCAN_THREADS + threadIdx.x];
  }
  const int64_t last = base + SCAN_TILE;
  if (threadIdx.x == 0 && last >= n && base < n + 1)
    out[n] = (block_offsets ? block_offsets[blockIdx.x] : 0ull) + total;
}

size_t scan_tmp_bytes(int64_t n) {
  size_t bytes = 0;
  int64_t m = n;
  while (m > SCAN_TILE) {
    m = ceil_div(m, SCAN_TILE);
    bytes += sizeof(uint64_t) * (size_t)(2 * m + 2);
  }
  return bytes + 256;
}

template <typename T>
static int exclusive_scan_impl(const T* in, uint64_t* out, int64_t n, void* tmp, cudaStream_t s) {
  if (n <= 0) {
    G500_CUDA(cudaMemsetAsync(out, 0, sizeof(uint64_t), s));
    return G500_OK;
  }
  int64_t nb = ceil_div(n, SCAN_TILE);
  if (nb == 1) {
    scan_tile_kernel<T><<<1, SCAN_THREADS, 0, s>>>(in, out, n, nullptr);
    G500_CUDA(cudaGetLastError());
    return G500_OK;
  }
  uint64_t* partial = reinterpret_cast<uint64_t*>(tmp);
  uint64_t* partial_scan = partial + nb + 1;
  void* rest = partial_scan + nb + 1;
  scan_reduce_kernel<T><<<(unsigned)nb, SCAN_THREADS, 0, s>>>(in, n, partial);
  G500_CUDA(cudaGetLastError());
  G500_TRY(exclusive_scan_impl<uint64_t>(partial, partial_scan, nb, rest, s));
  scan_tile_kernel<T><<<(unsigned)nb, SCAN_THREADS, 0, s>>>(in, out, n, partial_scan);
  G500_CUDA(cudaGetLastError());
  return G500_OK;
}

int exclusive_scan_u32(const uint32_t* in, uint64_t* out, int64_t n, void* tmp, cudaStream_t s) {
  return exclusive_scan_impl<uint32_t>(in, out, n, tmp, s);
}
int exclusive_scan_u64(const uint64_t* in, uint64_t* out, int64_t n, void* tmp, cudaStream_t s) {
  return exclusive_scan_impl<uint64_t>(in, out, n, tmp, s);
}

// ---------------------------------------------------------------------------
// LSD radix sort
//
// The bits are split evenly over ceil(bits / 9) passes of 8 or 9 bits (fewer
// where the whole key has fewer).  Per pass: digit counts per block
// (rs_upsweep_kernel), their exclusive scan in (digit, block) order, and the
// stable placement (rs_downsweep_kernel).  Each block owns a contiguous run of
// whole tiles.
//
// Memory-bound by design: a pass reads the keys twice and writes them once.  A
// tile is first put in digit order in shared memory, so that a warp's stores
// cover runs of one digit (8192 keys over 512 digits: 16 keys, 128 bytes on
// average); storing keys straight from the threads that ranked them wrote
// single 8-byte words all over the output.  Lanes with equal digits are found
// by one ballot per digit bit: __match_any_sync takes time per distinct value,
// which made uniform digits (the common case) twice as slow as skewed ones.
// 134 M edge keys at SCALE 22 (44 bits): six passes of 2.5-4 ms before, five of
// 0.9-1.1 ms now (counting 0.16, placing 0.76-0.90: 2.6 TB/s); 19.6 -> 5.0 ms.
// ---------------------------------------------------------------------------
constexpr int RS_THREADS = 512;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_ITEMS = 16;  // keys per lane per tile
constexpr int RS_TILE = RS_THREADS * RS_ITEMS;
constexpr int RS_MAX_BITS = 9;
constexpr int RS_MAX_BINS = 1 << RS_MAX_BITS;
static_assert(RS_MAX_BINS <= RS_THREADS, "one thread per digit");
static_assert(RS_TILE < 65536, "16-bit tile positions");

static int rs_num_blocks(int64_t n) {
  const int64_t tiles = ceil_div(n, RS_TILE);
  return (int)std::max<int64_t>(1, std::min<int64_t>(tiles, (int64_t)num_sms() * 2));
}

// Each block owns a contiguous run of whole tiles: [tile_begin, tile_end).
__device__ __forceinline__ void rs_block_range(int64_t n, int64_t* b, int64_t* e) {
  const int64_t tiles = (n + RS_TILE - 1) / RS_TILE;
  const int64_t t0 = tiles * blockIdx.x / gridDim.x, t1 = tiles * (blockIdx.x + 1) / gridDim.x;
  *b = min(n, t0 * RS_TILE);
  *e = min(n, t1 * RS_TILE);
}

// lanes whose digit equals this lane's
template <int BITS>
__device__ __forceinline__ unsigned rs_peers(unsigned d) {
  unsigned m = FULL_MASK;
#pragma unroll
  for (int b = 0; b < BITS; ++b) {
    const bool one = (d >> b) & 1u;
    const unsigned v = __ballot_sync(FULL_MASK, one);
    m &= one ? v : ~v;
  }
  return m;
}

// Digit counts of the block's keys.  Shared-memory atomics without a return
// value, in four copies by lane, so that the lanes of a warp that share a digit
// (row digits of a degree-sorted graph are mostly the smallest) meet on four
// addresses instead of one; counting them by ballots took 0.53 ms a pass for
// 134 M keys, this takes 0.16 (6.7 TB/s).
template <int BITS>
__global__ void __launch_bounds__(RS_THREADS) rs_upsweep_kernel(const uint64_t* __restrict__ keys, int64_t n,
                                                               int shift, unsigned mask,
                                                               uint32_t* __restrict__ hist /* [bins][grid] */) {
  constexpr int BINS = 1 << BITS;
  constexpr int COPIES = 4;
  __shared__ uint32_t wh[BINS * COPIES];
  for (int i = threadIdx.x; i < BINS * COPIES; i += RS_THREADS) wh[i] = 0;
  __syncthreads();
  int64_t b, e;
  rs_block_range(n, &b, &e);
  const unsigned copy = threadIdx.x & (COPIES - 1);
  constexpr int U = 8;  // keys in flight per thread
  for (int64_t base = b; base < e; base += RS_THREADS * U) {
    uint64_t k[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i = base + u * RS_THREADS + threadIdx.x;
      k[u] = i < e ? __ldcs(keys + i) : 0ull;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (base + u * RS_THREADS + threadIdx.x < e)
        atomicAdd(&wh[((unsigned)(k[u] >> shift) & mask) * COPIES + copy], 1u);
  }
  __syncthreads();
  for (int d = threadIdx.x; d < BINS; d += RS_THREADS) {
    uint32_t c = 0;
#pragma unroll
    for (int w = 0; w < COPIES; ++w) c += wh[d * COPIES + w];
    hist[(int64_t)d * gridDim.x + blockIdx.x] = c;
  }
}

template <int BITS>
struct RsShared {
  static constexpr int BINS = 1 << BITS;
  uint64_t keys[RS_TILE];           // the tile in digit order
  unsigned long long run[BINS];     // output position of the block's next key of each digit
  unsigned long long gofs[BINS];    // output position of a digit's tile keys, less their tile position
  uint32_t warp_sum[RS_WARPS];
  uint16_t wc[RS_WARPS][BINS];      // per-warp digit counts, then each warp's first tile position of the digit
};

template <int BITS>
__global__ void __launch_bounds__(RS_THREADS, 2) rs_downsweep_kernel(const uint64_t* __restrict__ keys,
                                                                    uint64_t* __restrict__ out, int64_t n, int shift,
                                                                    unsigned mask,
                                                                    const uint64_t* __restrict__ offsets) {
  constexpr int BINS = 1 << BITS;
  extern __shared__ __align__(16) unsigned char rs_raw[];
  RsShared<BITS>& sh = *reinterpret_cast<RsShared<BITS>*>(rs_raw);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int d = threadIdx.x; d < BINS; d += RS_THREADS) sh.run[d] = offsets[(int64_t)d * gridDim.x + blockIdx.x];
  int64_t b, e;
  rs_block_range(n, &b, &e);
  const unsigned lt_mask = (1u << lane) - 1u;
  for (int64_t tile = b; tile < e; tile += RS_TILE) {
    // keys of warp w: tile + w*512 + j*32 + lane, so (warp, j, lane) order is index order;
    // past the end all-ones keys, which sort to the tile's end and are not written
    const int64_t wbase = tile + (int64_t)warp * (RS_ITEMS * 32) + lane;
    uint64_t k[RS_ITEMS];
#pragma unroll
    for (int j = 0; j < RS_ITEMS; ++j) k[j] = wbase + j * 32 < e ? __ldcs(keys + wbase + j * 32) : ~0ull;
    for (int d = lane; d < BINS; d += 32) sh.wc[warp][d] = 0;
    __syncwarp();
    uint16_t rank[RS_ITEMS];
#pragma unroll
    for (int j = 0; j < RS_ITEMS; ++j) {
      const unsigned d = (unsigned)(k[j] >> shift) & mask;
      const unsigned peers = rs_peers<BITS>(d);
      const unsigned r = __popc(peers & lt_mask);
      const unsigned before = sh.wc[warp][d];
      __syncwarp();
      if (r == 0) sh.wc[warp][d] = (uint16_t)(before + __popc(peers));
      __syncwarp();
      rank[j] = (uint16_t)(before + r);
    }
    __syncthreads();
    // thread d: digit d's count over the warps, its first tile position, and each warp's
    uint32_t total = 0;
    if (threadIdx.x < BINS) {
#pragma unroll
      for (int w = 0; w < RS_WARPS; ++w) total += sh.wc[w][threadIdx.x];
    }
    uint32_t x = total;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(FULL_MASK, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) sh.warp_sum[warp] = x;
    __syncthreads();
    if (threadIdx.x < BINS) {
      uint32_t pos = x - total;
#pragma unroll
      for (int w = 0; w < RS_WARPS; ++w)
        if (w < warp) pos += sh.warp_sum[w];
      sh.gofs[threadIdx.x] = sh.run[threadIdx.x] - pos;
      sh.run[threadIdx.x] += total;
#pragma unroll
      for (int w = 0; w < RS_WARPS; ++w) {
        const uint32_t c = sh.wc[w][threadIdx.x];
        sh.wc[w][threadIdx.x] = (uint16_t)pos;
        pos += c;
      }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < RS_ITEMS; ++j) {
      const unsigned d = (unsigned)(k[j] >> shift) & mask;
      sh.keys[sh.wc[warp][d] + rank[j]] = k[j];
    }
    __syncthreads();
    const int count = (int)min((int64_t)RS_TILE, e - tile);
#pragma unroll
    for (int j = 0; j < RS_ITEMS; ++j) {
      const int i = j * RS_THREADS + threadIdx.x;
      if (i < count) {
        const uint64_t key = sh.keys[i];
        out[sh.gofs[(unsigned)(key >> shift) & mask] + i] = key;
      }
    }
    // the next tile touches keys and gofs only after its own barriers
  }
}

size_t sort_tmp_bytes(int64_t n) {
  const int g = rs_num_blocks(n);
  const size_t hist = sizeof(uint32_t) * (size_t)g * RS_MAX_BINS;
  const size_t offs = sizeof(uint64_t) * ((size_t)g * RS_MAX_BINS + 1);
  return hist + offs + scan_tmp_bytes((int64_t)g * RS_MAX_BINS) + 1024;
}

template <int BITS>
static int rs_pass(const uint64_t* src, uint64_t* dst, int64_t n, int shift, unsigned mask, int g, uint32_t* hist,
                   uint64_t* offs, void* scan_tmp, cudaStream_t s) {
  rs_upsweep_kernel<BITS><<<g, RS_THREADS, 0, s>>>(src, n, shift, mask, hist);
  G500_CUDA(cudaGetLastError());
  G500_TRY(exclusive_scan_u32(hist, offs, (int64_t)g * (1 << BITS), scan_tmp, s));
  G500_CUDA(cudaFuncSetAttribute(rs_downsweep_kernel<BITS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(RsShared<BITS>)));
  rs_downsweep_kernel<BITS><<<g, RS_THREADS, sizeof(RsShared<BITS>), s>>>(src, dst, n, shift, mask, offs);
  G500_CUDA(cudaGetLastError());
  return G500_OK;
}

int radix_sort_u64(uint64_t* keys, uint64_t* alt, int64_t n, int lo_bit, int hi_bit, void* tmp,
                   cudaStream_t s, uint64_t** result) {
  *result = keys;
  if (n <= 1 || hi_bit <= lo_bit) return G500_OK;
  const int g = rs_num_blocks(n);
  uint32_t* hist = reinterpret_cast<uint32_t*>(tmp);
  uint64_t* offs = reinterpret_cast<uint64_t*>(
      (reinterpret_cast<uintptr_t>(hist + (size_t)g * RS_MAX_BINS) + 255) & ~uintptr_t(255));
  void* scan_tmp = reinterpret_cast<void*>(
      (reinterpret_cast<uintptr_t>(offs + (size_t)g * RS_MAX_BINS + 1) + 255) & ~uintptr_t(255));
  uint64_t* src = keys;
  uint64_t* dst = alt;
  const int total = hi_bit - lo_bit;
  const int passes = (int)ceil_div(total, RS_MAX_BITS);
  for (int p = 0; p < passes; ++p) {
    const int b0 = total * p / passes, b1 = total * (p + 1) / passes;
    const int shift = lo_bit + b0, bits = b1 - b0;
    const unsigned mask = (1u << bits) - 1u;
    if (bits > 8) G500_TRY(rs_pass<9>(src, dst, n, shift, mask, g, hist, offs, scan_tmp, s));
    else G500_TRY(rs_pass<8>(src, dst, n, shift, mask, g, hist, offs, scan_tmp, s));
    std::swap(src, dst);
  }
  *result = src;
  return G500_OK;
}

}  // namespace g500
