// pred to a pageable host buffer for g500_bfs_run (the reference's driver
// allocates pred with plain host memory, main.cc:74-75): a kernel packs the
// int64 entries into 32 bits and stores them over PCIe into a pinned staging
// buffer itself, in chunks, marking each when it is complete; host threads,
// already waiting, expand a chunk into the caller's array while the next ones
// cross.  The runtime's own pageable copy goes through its staging buffers at
// about half the pinned rate, and a pack kernel followed by one copy and one
// event per chunk left the link idle between copies and the threads asleep until
// the first: a call with its search took 265 / 293 / 1090 / 850 us at SCALE 16 / 18 /
// 21 / 22 and takes 120 / 148 / 370 / 555.  A pinned pred keeps its single DMA
// copy.  The caller's array holds the same int64 values either way (bfs.hpp:1203,
// :2470 encoding: parent | level << 48, -1 unreached).
//
// Graphs with more than 2^PACK_BITS ids, and runs with a level over
// PACK_MAX_LEVEL, copy the int64 entries instead (packed_entry.h).
#include "g500_internal.cuh"
#include "pred_expander.h"

#include <algorithm>
#include <vector>

namespace g500 {
namespace {

// Chunks of at least 512 KB of packed entries (a chunk's fences and mark cost
// about 5 us: with 16 chunks whatever the size a SCALE 18 call took 200 us
// instead of 153), at most 16.
constexpr int PRED_CHUNKS = 16;
constexpr int64_t CHUNK_ENTRIES = 1 << 17;
inline int chunks_for(int64_t n) {
  int c = 1;
  while (c < PRED_CHUNKS && n / (2 * c) >= CHUNK_ENTRIES) c *= 2;
  return c;
}
constexpr int PACK_GROUPS = 2;     // groups of blocks, on alternate chunks: one packs while the other's stores drain
constexpr int PACK_BLOCKS = 64;    // blocks per group
constexpr int PACK_THREADS = 256;

// Device state of the packing: blocks that have finished a chunk, and whether
// any entry did not fit.  Left clear by every run but one with such an entry.
struct PackState {
  unsigned done[PRED_CHUNKS];
  unsigned bad;
};

// The chunks' marks, in pinned memory behind the packed entries.
struct PackTail {
  volatile uint32_t ready[PRED_CHUNKS];  // run number << 1 | an entry so far did not fit
};

// Chunk c holds entries [c, c + 1) * n / nchunks (n is a multiple of 65536).
// A chunk is marked by the last block of its group, after every block's stores
// have reached host memory (system-wide fences).  A search too deep for the
// entries (the last level it ran found nothing) is marked so at once, and
// nothing is sent or expanded: 16 threads that expand most of it before the copy
// of the int64 entries into the same memory took 2.2 ms longer at 2^21 ids.
__global__ void __launch_bounds__(PACK_THREADS) pack_to_host_kernel(const int64_t* __restrict__ pred, int64_t n,
                                                                    int nchunks, uint32_t* __restrict__ out,
                                                                    const BfsCtl* __restrict__ ctl, PackState* st,
                                                                    volatile uint32_t* ready, uint32_t run) {
  if (ctl->root_has_edges && ctl->num_levels > (unsigned)PACK_MAX_LEVEL + 1) {
    if (blockIdx.x == 0 && threadIdx.x < nchunks) ready[threadIdx.x] = run << 1 | 1u;
    return;
  }
  const int group = blockIdx.x % PACK_GROUPS;
  const int64_t rank = blockIdx.x / PACK_GROUPS;
  const int64_t len = n / nchunks;
  for (int c = group; c < nchunks; c += PACK_GROUPS) {
    bool bad = false;
    for (int64_t i = c * len + (rank * PACK_THREADS + threadIdx.x) * 4; i < (c + 1) * len;
         i += (int64_t)PACK_BLOCKS * PACK_THREADS * 4) {
      const longlong2 a = __ldcs(reinterpret_cast<const longlong2*>(pred + i));
      const longlong2 b = __ldcs(reinterpret_cast<const longlong2*>(pred + i + 2));
      const long long x[4] = {a.x, a.y, b.x, b.y};
      uint32_t e[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (x[k] == -1) {
          e[k] = PACK_NONE;
        } else {
          const uint64_t parent = (uint64_t)x[k] & ((1ull << 48) - 1);
          const uint64_t level = (uint64_t)x[k] >> 48;
          bad |= parent >= (1ull << PACK_BITS) || level > (uint64_t)PACK_MAX_LEVEL;
          e[k] = (uint32_t)parent | ((uint32_t)level << PACK_BITS);
        }
      }
      *reinterpret_cast<uint4*>(out + i) = make_uint4(e[0], e[1], e[2], e[3]);
    }
    if (bad) atomicOr(&st->bad, 1u);
    __threadfence_system();
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(&st->done[c], 1u) + 1 == PACK_BLOCKS) {
      __threadfence_system();
      st->done[c] = 0;
      ready[c] = run << 1 | (atomicOr(&st->bad, 0u) ? 1u : 0u);
    }
  }
}

}  // namespace

void pred_expander_free(g500_bfs* b) {
  delete b->expander;
  b->expander = nullptr;
  dev_free(b->d_pack_state);
  b->d_pack_state = nullptr;
  if (b->h_pack) cudaFreeHost(b->h_pack);
  b->h_pack = nullptr;
}

int pred_to_host_packed(g500_bfs* b, int64_t* host_pred, cudaStream_t s, bool* packed) {
  g500_graph* g = b->g;
  *packed = false;
  const int64_t n = g->nolv;
  if (n > (1ll << PACK_BITS) || n % (4 * PRED_CHUNKS) != 0 || b->pack_host_off) return G500_OK;
  cudaPointerAttributes attr;
  if (cudaPointerGetAttributes(&attr, host_pred) != cudaSuccess) {
    cudaGetLastError();  // not a pointer the runtime knows: pageable
    attr.type = cudaMemoryTypeUnregistered;
  }
  if (attr.type != cudaMemoryTypeUnregistered) return G500_OK;  // pinned (or device): one DMA copy is faster
  if (!b->expander) {
    void* st = b->d_pack_state;
    if (!st) G500_TRY(dev_alloc(&st, sizeof(PackState), "pred packing state"));
    b->d_pack_state = st;
    G500_CUDA(cudaMemsetAsync(st, 0, sizeof(PackState), s));
    if (!b->h_pack) {
      G500_CUDA(cudaHostAlloc(&b->h_pack, sizeof(uint32_t) * (size_t)n + sizeof(PackTail), cudaHostAllocDefault));
      memset(b->h_pack + n, 0, sizeof(PackTail));
    }
    const int hw = (int)std::thread::hardware_concurrency();
    b->expander = new PredExpander(std::max(1, std::min(hw > 0 ? hw : 1, 16)));
  }
  PackState* st = static_cast<PackState*>(b->d_pack_state);
  PackTail* tail = reinterpret_cast<PackTail*>(b->h_pack + n);
  G500_CUDA(cudaMemcpyAsync(b->h_ctl, b->d_ctl, sizeof(BfsCtl), cudaMemcpyDeviceToHost, s));
  const uint32_t run = ++b->pack_run & 0x7FFFFFFFu;
  pack_to_host_kernel<<<PACK_GROUPS * PACK_BLOCKS, PACK_THREADS, 0, s>>>(b->d_pred, n, chunks_for(n), b->h_pack,
                                                                         b->d_ctl, st, tail->ready, run);
  G500_CUDA(cudaGetLastError());
  const auto state = [s] {
    const cudaError_t e = cudaStreamQuery(s);
    if (e == cudaSuccess) return WorkState::complete;
    if (e == cudaErrorNotReady) return WorkState::running;
    cudaGetLastError();
    return WorkState::refused;
  };
  const bool complete = b->expander->run(b->h_pack, host_pred, n, chunks_for(n), tail->ready, run, state);
  G500_CUDA(cudaStreamSynchronize(s));
  if (!complete) return set_error(G500_E_DEVICE, "the packed pred did not arrive");
  bool bad = false;
  for (int c = 0; c < chunks_for(n); ++c) bad |= tail->ready[c] & 1u;
  if (bad) {  // a level or an id beyond the packed fields: the caller gets the int64 copy instead
    G500_CUDA(cudaMemsetAsync(st, 0, sizeof(PackState), s));
    return G500_OK;
  }
  *packed = true;
  return G500_OK;
}

}  // namespace g500
