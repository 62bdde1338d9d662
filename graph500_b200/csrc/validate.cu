// Graph500 result validation on the device: BfsValidation::validate
// (mpi/validate.hpp:506-802) for one rank.
//
//   vertex pass  -- check_value_ranges (:822-839), root is its own parent
//                   (:529-537), no other self parent (:542-571), and
//                   check_bfs_depth_map_using_predecessors (:920-995)
//   edge pass    -- every input edge: both ends in or both out of the tree,
//                   |depth difference| <= 1, count edge_visit_count, and mark
//                   vertices whose parent edge appears (:598-776)
//   parent pass  -- every reached non-root vertex has an input edge to its
//                   parent (:780-792)
//
// The reference stops after the first failing stage; this version computes
// every stage (guarding the reads an out-of-range parent would make) and
// reports per-stage error counts.  The result is valid iff all are zero.
#include "g500_internal.cuh"

#include <algorithm>
#include <mutex>

namespace g500 {

// VE_UNPACKED: entries that do not fit the packed form below (a flag, no error)
enum { VE_RANGE, VE_ROOT, VE_SELF, VE_DEPTH, VE_EDGE, VE_MISSING, VE_COUNT_EDGES, VE_UNPACKED, VE_N };

// Packed entries (packed_entry.h) for graphs of at most 2^PACK_BITS vertex ids
// and depths of at most PACK_MAX_LEVEL.  The edge pass reads two entries per
// input edge at random, so their size decides how many come from L2 (SCALE 24:
// 67 MB instead of 134 MB).
constexpr int VAL_VERTS = 4;  // vertices per thread in flight (vertex and parent passes: 86 / 81 us at SCALE 24 with one)

__device__ __forceinline__ int64_t pred_of(int64_t e) { return (int64_t)((uint64_t)e << 16) >> 16; }  // :809
__device__ __forceinline__ int depth_of(int64_t e) { return (int)((e >> 48) & 0xFFFF); }              // :813

__device__ __forceinline__ void warp_add(unsigned long long* dst, unsigned long long v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(FULL_MASK, v, o);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd(dst, v);
}

// pack: null, or the packed entries to write; entries that do not fit raise
// VE_UNPACKED, and the later passes then read pred itself.
__global__ void __launch_bounds__(256) val_vertex_kernel(const int64_t* __restrict__ pred, int64_t nlocal,
                                                         int64_t nglobal, int64_t root, uint32_t* __restrict__ pack,
                                                         unsigned long long* err) {
  uint32_t range = 0, self = 0, depth = 0;  // per thread: far fewer than 2^32
  bool unpacked = false;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < nlocal; i0 += nthreads * VAL_VERTS) {
    int64_t e[VAL_VERTS], parent[VAL_VERTS];
    bool look[VAL_VERTS];  // the parent's entry is read, all of them in flight together
#pragma unroll
    for (int u = 0; u < VAL_VERTS; ++u) {
      const int64_t i = i0 + u * nthreads;
      e[u] = i < nlocal ? pred[i] : -1;
    }
#pragma unroll
    for (int u = 0; u < VAL_VERTS; ++u) {
      const int64_t i = i0 + u * nthreads, p = pred_of(e[u]);
      look[u] = i < nlocal && p >= 0 && p < nglobal && i != root;  // nglobal <= nlocal
      parent[u] = look[u] ? pred[p] : 0;
    }
#pragma unroll
    for (int u = 0; u < VAL_VERTS; ++u) {
      const int64_t i = i0 + u * nthreads, p = pred_of(e[u]);
      const int d = depth_of(e[u]);
      if (i >= nlocal) continue;
      if (pack) {
        const bool none = p == -1 && d == 0xFFFF;
        unpacked |= !none && (p < 0 || p > (int64_t)PACK_ID || d > PACK_MAX_LEVEL);
        pack[i] = none ? PACK_NONE : (uint32_t)p | ((uint32_t)d << PACK_BITS);
      }
      if (p < -1 || p >= nglobal) {
        ++range;
        continue;
      }
      if (i != root && p != -1 && p == i) ++self;
      if (p == -1 && d != 0xFFFF) ++depth;
      else if (p != -1 && d == 0xFFFF) ++depth;
      if (look[u]) {
        if (depth_of(parent[u]) == 0xFFFF) ++depth;
        if (d != depth_of(parent[u]) + 1) ++depth;
      }
    }
  }
  warp_add(&err[VE_RANGE], range);
  warp_add(&err[VE_SELF], self);
  warp_add(&err[VE_DEPTH], depth);
  warp_add(&err[VE_UNPACKED], unpacked);
}

// validate.hpp:513-515 only reports a root outside [0, nglobalverts); its
// pred entry then fails the range check.  A root outside pred[] is refused.
__global__ void val_root_kernel(const int64_t* __restrict__ pred, int64_t root, int64_t nlocal,
                                unsigned long long* err) {
  if (root < 0 || root >= nlocal) {
    atomicAdd(&err[VE_ROOT], 1ull);
    return;
  }
  const int64_t e = pred[root];
  if (pred_of(e) != root) atomicAdd(&err[VE_ROOT], 1ull);
  if (depth_of(e) != 0) atomicAdd(&err[VE_DEPTH], 1ull);
}

__device__ __forceinline__ int64_t ev0(const g500_packed_edge& e) {
  return (int64_t)e.v0_low | ((int64_t)(e.high & 0xFFFF) << 32);
}
__device__ __forceinline__ int64_t ev1(const g500_packed_edge& e) {
  return (int64_t)e.v1_low | ((int64_t)(e.high >> 16) << 32);
}

// One edge against its ends' entries.
struct EdgeCheck {
  uint32_t bad = 0, count = 0;  // per thread: far fewer than 2^32
  __device__ __forceinline__ void full(int64_t src, int64_t tgt, int64_t ps, int64_t pt, uint8_t* valid) {
    const int sd = depth_of(ps), td = depth_of(pt);
    if (sd != 0xFFFF && td == 0xFFFF) ++bad;
    else if (sd == 0xFFFF && td != 0xFFFF) ++bad;
    else if (sd - td < -1 || sd - td > 1) ++bad;
    else if (sd != 0xFFFF) ++count;
    if (pred_of(ps) == tgt) valid[src] = 1;
    if (pred_of(pt) == src) valid[tgt] = 1;
  }
  // the same from packed entries: two unreached ends are neither bad nor counted
  __device__ __forceinline__ void packed(uint32_t src, uint32_t tgt, uint32_t ps, uint32_t pt, uint8_t* valid) {
    if (ps == PACK_NONE || pt == PACK_NONE) {
      bad += ps != pt;
    } else {
      const int diff = (int)(ps >> PACK_BITS) - (int)(pt >> PACK_BITS);
      if (diff < -1 || diff > 1) ++bad;
      else ++count;
    }
    if (ps != PACK_NONE && (ps & PACK_ID) == tgt) valid[src] = 1;
    if (pt != PACK_NONE && (pt & PACK_ID) == src) valid[tgt] = 1;
  }
};

// Bound by the random reads of the ends' entries (two per edge).  pack: the
// packed entries, or null; used when every entry fitted.  U edges per thread, their
// reads in flight together (four as three 16-byte loads where the list is aligned
// to that).  What pays depends on where the entries lie (see val_packs).
template <int U>
__global__ void __launch_bounds__(256) val_edge_kernel(const g500_packed_edge* __restrict__ edges, int64_t m,
                                                       const int64_t* __restrict__ pred,
                                                       const uint32_t* __restrict__ pack, int64_t nlocal,
                                                       uint8_t* valid, unsigned long long* err) {
  const bool use_pack = pack && *(volatile unsigned long long*)&err[VE_UNPACKED] == 0;
  const bool wide = (reinterpret_cast<uintptr_t>(edges) & 15) == 0;
  EdgeCheck c;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * U; i0 < m;
       i0 += nthreads * U) {
    g500_packed_edge ed[U];
    const int n = (int)min((int64_t)U, m - i0);
    if (U == 4 && wide && n == U) {  // i0 is a multiple of 4 edges: 48 bytes
      const uint4* q = reinterpret_cast<const uint4*>(edges + i0);
      const uint4 a = __ldcs(q), b = __ldcs(q + 1), d = __ldcs(q + 2);
      ed[0] = {a.x, a.y, a.z};
      ed[1 % U] = {a.w, b.x, b.y};
      ed[2 % U] = {b.z, b.w, d.x};
      ed[3 % U] = {d.y, d.z, d.w};
    } else {
#pragma unroll
      for (int u = 0; u < U; ++u) ed[u] = u < n ? edges[i0 + u] : edges[i0];
    }
    bool in[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      in[u] = u < n && ev0(ed[u]) < nlocal && ev1(ed[u]) < nlocal;
      c.bad += u < n && !in[u];
    }
    if (use_pack) {
      uint32_t ps[U], pt[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        ps[u] = in[u] ? __ldg(pack + ed[u].v0_low) : PACK_NONE;
        pt[u] = in[u] ? __ldg(pack + ed[u].v1_low) : PACK_NONE;
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (in[u]) c.packed(ed[u].v0_low, ed[u].v1_low, ps[u], pt[u], valid);
    } else {
      int64_t ps[U], pt[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        ps[u] = in[u] ? pred[ev0(ed[u])] : 0;
        pt[u] = in[u] ? pred[ev1(ed[u])] : 0;
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (in[u]) c.full(ev0(ed[u]), ev1(ed[u]), ps[u], pt[u], valid);
    }
  }
  warp_add(&err[VE_EDGE], c.bad);
  warp_add(&err[VE_COUNT_EDGES], c.count);
}

__global__ void __launch_bounds__(256) val_parent_kernel(const int64_t* __restrict__ pred,
                                                         const uint32_t* __restrict__ pack, int64_t nlocal,
                                                         int64_t root, const uint8_t* __restrict__ valid,
                                                         unsigned long long* err) {
  const bool use_pack = pack && *(volatile unsigned long long*)&err[VE_UNPACKED] == 0;
  uint32_t missing = 0;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < nlocal; i0 += nthreads * VAL_VERTS) {
    bool reached[VAL_VERTS], ok[VAL_VERTS];
#pragma unroll
    for (int u = 0; u < VAL_VERTS; ++u) {
      const int64_t i = i0 + u * nthreads;
      reached[u] = i < nlocal && i != root && (use_pack ? pack[i] != PACK_NONE : pred_of(pred[i]) != -1);
      ok[u] = i < nlocal && valid[i];
    }
#pragma unroll
    for (int u = 0; u < VAL_VERTS; ++u) missing += reached[u] && !ok[u];
  }
  warp_add(&err[VE_MISSING], missing);
}

// Whether the entries are packed for the edge pass, and how many edges a thread
// takes there.  Up to 2^20 ids the 64-bit entries stay in L2; up to 2^19 more threads
// with one edge each hide their latency best: a validation at SCALE 16 / 17 / 18 takes
// 67 / 68 / 82 us so, 81 / 94 / 107 from packed entries by four edges and 81 / 83 / 102
// by two; at SCALE 20 64-bit entries take 182 us by four edges and 190 by one, packed
// ones 196 and 206.  Above, packed entries halve what is read, two edges a thread up to
// 2^23 ids (SCALE 21 / 23 327 / 1164 us, four 327 / 1162, one 340 / 1179), four beyond
// (SCALE 24 2381 us, two 2478, one 2520).  64-bit entries without the memory for
// packed ones, SCALE 22: 567 us by four edges, 592 by one.
static bool val_packs(int64_t nlocal) {
  return nlocal > int64_t(1) << 20 && nlocal <= int64_t(1) << PACK_BITS;
}
static int val_edges(bool packed, int64_t nlocal) {
  if (packed) return nlocal <= int64_t(1) << 23 ? 2 : 4;
  return nlocal <= int64_t(1) << 19 ? 1 : 4;
}

// The three passes over a result (the root's check and the counters' clearing apart).
static void val_passes(const g500_packed_edge* edges, int64_t m, const int64_t* pred, uint32_t* pack, int64_t nlocal,
                       int64_t nglobal, int64_t root, uint8_t* valid, unsigned long long* err, cudaStream_t s) {
  const int64_t most = (int64_t)num_sms() * 16;
  const unsigned vgrid = (unsigned)std::min<int64_t>(ceil_div(nlocal, 256), most);
  const unsigned egrid = (unsigned)std::min<int64_t>(ceil_div(m, 256), most);
  val_vertex_kernel<<<vgrid, 256, 0, s>>>(pred, nlocal, nglobal, root, pack, err);
  const int per = val_edges(pack != nullptr, nlocal);
  if (m > 0) {
    if (per == 1) val_edge_kernel<1><<<egrid, 256, 0, s>>>(edges, m, pred, pack, nlocal, valid, err);
    else if (per == 2) val_edge_kernel<2><<<egrid, 256, 0, s>>>(edges, m, pred, pack, nlocal, valid, err);
    else val_edge_kernel<4><<<egrid, 256, 0, s>>>(edges, m, pred, pack, nlocal, valid, err);
  }
  val_parent_kernel<<<vgrid, 256, 0, s>>>(pred, pack, nlocal, root, valid, err);
}

// A call's scratch, given back to the graph at its end (or freed, where another
// call has given back its own in the meantime).
struct KeptScratch {
  g500_graph* g;
  void* p;
  size_t bytes;
  bool keep = true;
  ~KeptScratch() {
    void* none = nullptr;
    if (!p) return;
    if (keep && g->d_val.compare_exchange_strong(none, p)) g->val_bytes.store((int64_t)bytes);
    else dev_free(p);
  }
};

}  // namespace g500

using namespace g500;

extern "C" int g500_validate(g500_graph* g, const g500_packed_edge* edges, int64_t m, int edges_on_device,
                             int64_t root, const int64_t* pred, int pred_on_device, int64_t* edge_visit_count,
                             int* ok, g500_validate_report* report) {
  if (!g || !pred || !ok) return set_error(G500_E_INVAL, "null argument");
  if (!edges) {
    if (!g->d_edges) return set_error(G500_E_STATE, "graph keeps no edge list; pass one");
    edges = g->d_edges;
    m = g->num_edges;
    edges_on_device = 1;
  }
  G500_CUDA(cudaSetDevice(g->device));
  cudaStream_t s = g->stream;
  const int64_t nlocal = g->nolv;
  const int64_t nglobal = g->max_used_vertex + 1;  // main.cc:129-133
  std::vector<void*> owned;
  auto cleanup = [&]() {
    for (void* p : owned) dev_free(p);
  };
  const int64_t* d_pred = pred;
  const g500_packed_edge* d_edges = edges;
  int st = G500_OK;
  if (!pred_on_device) {
    int64_t* p = nullptr;
    st = dev_alloc_n(&p, nlocal, "validation pred copy");
    if (st != G500_OK) return st;
    owned.push_back(p);
    cudaError_t e = cudaMemcpyAsync(p, pred, sizeof(int64_t) * nlocal, cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) { cleanup(); return cuda_error(e, "cudaMemcpyAsync(pred)", __FILE__, __LINE__); }
    d_pred = p;
  }
  if (!edges_on_device && m > 0) {
    g500_packed_edge* p = nullptr;
    st = dev_alloc_n(&p, m, "validation edge copy");
    if (st != G500_OK) { cleanup(); return st; }
    owned.push_back(p);
    cudaError_t e = cudaMemcpyAsync(p, edges, sizeof(g500_packed_edge) * m, cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) { cleanup(); return cuda_error(e, "cudaMemcpyAsync(edges)", __FILE__, __LINE__); }
    d_edges = p;
  }
  // The scratch stays with the graph: allocating and freeing it took 0.7 ms per
  // call.  A call takes it out while it runs, so that another thread's call on
  // the same graph finds none and allocates its own.
  unsigned long long* d_err = nullptr;
  uint8_t* d_valid = nullptr;
  Slab scratch;
  scratch.add(&d_err, VE_N);
  scratch.add(&d_valid, nlocal);
  Slab small = scratch;
  uint32_t* d_pack = nullptr;  // packed entries, where the ids allow them
  const bool can_pack = val_packs(nlocal);
  if (can_pack) scratch.add(&d_pack, nlocal);
  KeptScratch kept{g, g->d_val.exchange(nullptr), scratch.bytes};
  if (kept.p) scratch.place(kept.p);
  else st = scratch.alloc(&kept.p, "validation scratch");
  if (st == G500_E_NOMEM && can_pack) {  // a fifth of the memory does without packed entries, for this call
    st = small.alloc(&kept.p, "validation scratch");
    kept.keep = false;
  }
  if (st != G500_OK) { cleanup(); return st; }
  cudaError_t e = cudaMemsetAsync(d_err, 0, sizeof(unsigned long long) * VE_N, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(d_valid, 0, (size_t)nlocal, s);
  if (e != cudaSuccess) { cleanup(); return cuda_error(e, "cudaMemsetAsync", __FILE__, __LINE__); }
  val_root_kernel<<<1, 1, 0, s>>>(d_pred, root, nlocal, d_err);
  val_passes(d_edges, m, d_pred, d_pack, nlocal, nglobal, root, d_valid, d_err, s);
  e = cudaGetLastError();
  unsigned long long h[VE_N];
  if (e == cudaSuccess) e = cudaMemcpyAsync(h, d_err, sizeof(h), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  cleanup();
  if (e != cudaSuccess) return cuda_error(e, "validation", __FILE__, __LINE__);
  g500_validate_report r;
  r.range_errors = (int64_t)h[VE_RANGE];
  r.root_errors = (int64_t)h[VE_ROOT];
  r.self_parent_errors = (int64_t)h[VE_SELF];
  r.depth_errors = (int64_t)h[VE_DEPTH];
  r.edge_errors = (int64_t)h[VE_EDGE];
  r.missing_parent_edge_errors = (int64_t)h[VE_MISSING];
  const bool valid = !(r.range_errors || r.root_errors || r.self_parent_errors || r.depth_errors ||
                       r.edge_errors || r.missing_parent_edge_errors);
  *ok = valid ? 1 : 0;
  if (edge_visit_count) *edge_visit_count = valid ? (int64_t)h[VE_COUNT_EDGES] : 0;
  if (report) *report = r;
  return G500_OK;
}

// ---------------------------------------------------------------------------
// Validation that allocates nothing.
//
// Some callers cannot call cudaMalloc: a host framework that owns all device
// memory through its own arena or caching allocator, or a serving loop that
// forbids allocation once it has started.  For them the scratch of the
// validator (one flag byte per vertex and the error counters) lives in
// file-scope device arrays of a fixed size, held by every GPU that loads the
// library until the process exits.  Host code cannot use the arrays' names as
// device addresses, so each device's addresses are fetched once with
// cudaGetSymbolAddress, with that device current.
// ---------------------------------------------------------------------------
namespace g500 {

static __device__ __align__(256) uint8_t g_static_valid[G500_VALIDATE_STATIC_MAX_VERTS];
static __device__ __align__(256) unsigned long long g_static_err[VE_N];

struct StaticScratch {
  uint8_t* valid = nullptr;
  unsigned long long* err = nullptr;
};
static StaticScratch g_static_scratch[64];
static std::mutex g_static_mu;

// G500_OK when p is device (or managed) memory of device dev.
static int on_device(const void* p, int dev, const char* what) {
  cudaPointerAttributes a;
  const cudaError_t e = cudaPointerGetAttributes(&a, p);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return set_error(G500_E_INVAL, "%s: not a CUDA pointer (%s)", what, cudaGetErrorString(e));
  }
  if (a.type != cudaMemoryTypeDevice && a.type != cudaMemoryTypeManaged)
    return set_error(G500_E_INVAL, "%s is not in device memory", what);
  if (a.type == cudaMemoryTypeDevice && a.device != dev)
    return set_error(G500_E_INVAL, "%s is on device %d, but device %d is current; make the device that holds the "
                     "buffers current before the call", what, a.device, dev);
  return G500_OK;
}

// Resolve this device's scratch addresses (first call on a device only).
static int static_scratch(int dev, StaticScratch* out) {
  if (dev < 0 || dev >= 64) return set_error(G500_E_INVAL, "device %d out of range", dev);
  std::lock_guard<std::mutex> lk(g_static_mu);
  StaticScratch& s = g_static_scratch[dev];
  if (!s.valid) {
    void* v = nullptr;
    void* e = nullptr;
    G500_CUDA(cudaGetSymbolAddress(&v, g_static_valid));
    G500_CUDA(cudaGetSymbolAddress(&e, g_static_err));
    s.valid = static_cast<uint8_t*>(v);
    s.err = static_cast<unsigned long long*>(e);
  }
  *out = s;
  return G500_OK;
}

}  // namespace g500

extern "C" int g500_validate_noalloc(const g500_packed_edge* dev_edges, int64_t num_edges, int64_t nglobalverts,
                                     int64_t nlocalverts, int64_t root, const int64_t* dev_pred, void* stream,
                                     int64_t* edge_visit_count, int* ok, g500_validate_report* report) {
  if (!dev_pred || !ok || (num_edges > 0 && !dev_edges)) return set_error(G500_E_INVAL, "null argument");
  if (num_edges < 0 || nlocalverts <= 0 || nglobalverts < 0 || nglobalverts > nlocalverts)
    return set_error(G500_E_INVAL, "bad sizes (num_edges %lld, nglobalverts %lld, nlocalverts %lld)",
                     (long long)num_edges, (long long)nglobalverts, (long long)nlocalverts);
  if (nlocalverts > G500_VALIDATE_STATIC_MAX_VERTS)
    return set_error(G500_E_RANGE, "g500_validate_noalloc handles at most %d vertices (pred_size %lld); "
                     "use g500_validate", G500_VALIDATE_STATIC_MAX_VERTS, (long long)nlocalverts);
  int dev = 0;
  G500_CUDA(cudaGetDevice(&dev));
  // the scratch and the kernels belong to the current device: pred and the
  // edge list must live there too (a peer's or a host pointer is refused)
  G500_TRY(on_device(dev_pred, dev, "pred"));
  if (num_edges > 0) G500_TRY(on_device(dev_edges, dev, "edge list"));
  StaticScratch sc;
  G500_TRY(static_scratch(dev, &sc));
  cudaStream_t s = (cudaStream_t)stream;
  // the arrays keep the last call's contents: clear what must start at zero
  G500_CUDA(cudaMemsetAsync(sc.err, 0, sizeof(unsigned long long) * VE_N, s));
  G500_CUDA(cudaMemsetAsync(sc.valid, 0, (size_t)nlocalverts, s));
  val_root_kernel<<<1, 1, 0, s>>>(dev_pred, root, nlocalverts, sc.err);
  val_passes(dev_edges, num_edges, dev_pred, nullptr, nlocalverts, nglobalverts, root, sc.valid, sc.err, s);
  G500_CUDA(cudaGetLastError());
  unsigned long long h[VE_N];
  G500_CUDA(cudaMemcpyAsync(h, sc.err, sizeof(h), cudaMemcpyDeviceToHost, s));
  G500_CUDA(cudaStreamSynchronize(s));
  g500_validate_report r;
  r.range_errors = (int64_t)h[VE_RANGE];
  r.root_errors = (int64_t)h[VE_ROOT];
  r.self_parent_errors = (int64_t)h[VE_SELF];
  r.depth_errors = (int64_t)h[VE_DEPTH];
  r.edge_errors = (int64_t)h[VE_EDGE];
  r.missing_parent_edge_errors = (int64_t)h[VE_MISSING];
  const bool valid = !(r.range_errors || r.root_errors || r.self_parent_errors || r.depth_errors ||
                       r.edge_errors || r.missing_parent_edge_errors);
  *ok = valid ? 1 : 0;
  if (edge_visit_count) *edge_visit_count = valid ? (int64_t)h[VE_COUNT_EDGES] : 0;
  if (report) *report = r;
  return G500_OK;
}
