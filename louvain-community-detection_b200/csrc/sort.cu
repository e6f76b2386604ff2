// sort.cu -- stable device radix sort, and the two ingest / output steps
// built on it: the CSR of an edge list and the community listing.
//
// Reference counterparts (upicine/louvain-community-detection):
//   parseGraph's CSR construction ........ utils.cu:168-229 (host, one
//                                          vector per row, file order)
//   printCommunities's grouping ........... utils.cu:270-293 (host, one
//                                          scan over init_comm per community)
//
// Radix sort: least-significant digit first, digits of at most 8 bits spread
// evenly over the key bits in use (21 bits: three passes of 7).  A pass is
// three launches over tiles of 4096 keys: a per-tile digit histogram (stored
// digit-major, so one exclusive scan of the whole table gives every (digit,
// tile) its output offset), the scan, and a scatter.  The scatter holds a
// tile in registers: each warp ranks its 256 keys round by round (equal
// digits of a round found with one ballot per digit bit), so the order of
// equal keys is kept, then the tile is reordered by digit in shared memory
// and written out in runs.  The first pass reads its keys and payload from a
// source (an edge list, an index), the last one writes the payload where the
// caller wants it: no separate expand or gather pass.
#include <algorithm>
#include <mutex>

#include "lv_internal.h"

namespace lvb {
namespace {

constexpr int kSortThreads = 512;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortItems = 8;                            // keys per thread
constexpr uint32_t kSortTile = kSortThreads * kSortItems;  // 4096
constexpr uint32_t kWarpKeys = kSortTile / kSortWarps;     // 256 per warp
constexpr int kRadix = 256;

// Keys j .. j + 3 (j a multiple of 4) with 128-bit loads where the array
// allows them: scratch always does, a caller's array may start anywhere.
template <typename K>
__device__ __forceinline__ void load4(const K* __restrict__ a, uint64_t j, K (&k)[4]) {
  if (((uintptr_t)a & 15u) == 0) {
    constexpr int kVec = (int)(16 / sizeof(K));
#pragma unroll
    for (int i = 0; i < 4; i += kVec) {
      const uint4 x = *reinterpret_cast<const uint4*>(a + j + i);
      if constexpr (sizeof(K) == 4) {
        k[0] = x.x;
        k[1] = x.y;
        k[2] = x.z;
        k[3] = x.w;
      } else {
        k[i] = (K)x.x | ((K)x.y << 32);
        k[i + 1] = (K)x.z | ((K)x.w << 32);
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < 4; i++) k[i] = a[j + i];
  }
}

// Where a pass reads entry j: its key (key4: four keys from a multiple of
// 4), and its payload words.
template <typename K, int NP>
struct ArraySource {
  const K* __restrict__ keys;
  const uint32_t* __restrict__ p[NP];
  __device__ __forceinline__ K key(uint64_t j) const { return keys[j]; }
  __device__ __forceinline__ void key4(uint64_t j, K (&k)[4]) const { load4(keys, j, k); }
  __device__ __forceinline__ uint32_t pay(uint64_t j, int q) const { return p[q][j]; }
};
// Keys in an array, the payload is the index itself.
template <typename K>
struct IndexSource {
  const K* __restrict__ keys;
  __device__ __forceinline__ K key(uint64_t j) const { return keys[j]; }
  __device__ __forceinline__ void key4(uint64_t j, K (&k)[4]) const { load4(keys, j, k); }
  __device__ __forceinline__ uint32_t pay(uint64_t j, int) const { return (uint32_t)j; }
};
// Directed entries of an edge list in the order the reference reader appends
// them (utils.cu:302-313): edge e gives entry 2e in row src[e] and, unless it
// is a self-loop, entry 2e+1 in row dst[e]; a self-loop's second entry gets
// the key n and sorts after every row.  Payload: the entry's column and
// weight (|w| as utils.cu:295; 1 without a weight array).
struct EdgeSource {
  const uint32_t* __restrict__ src;
  const uint32_t* __restrict__ dst;
  const float* __restrict__ w;
  uint32_t n;
  uint32_t* bad;  // set when an index is >= n
  __device__ __forceinline__ uint32_t key(uint64_t j) const {
    const uint32_t a = src[j >> 1], b = dst[j >> 1];
    return (j & 1u) ? second(a, b) : first(a, b);
  }
  __device__ __forceinline__ void key4(uint64_t j, uint32_t (&k)[4]) const {
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const uint32_t a = src[(j >> 1) + i], b = dst[(j >> 1) + i];
      k[2 * i] = first(a, b);
      k[2 * i + 1] = second(a, b);
    }
  }
  __device__ __forceinline__ uint32_t first(uint32_t a, uint32_t b) const {
    if (a >= n || b >= n) atomicExch(bad, 1u);
    return a < n ? a : n;
  }
  __device__ __forceinline__ uint32_t second(uint32_t a, uint32_t b) const {
    return (a != b && b < n) ? b : n;
  }
  __device__ __forceinline__ uint32_t pay(uint64_t j, int q) const {
    if (q == 0) return (j & 1u) ? src[j >> 1] : dst[j >> 1];
    return __float_as_uint(w ? fabsf(w[j >> 1]) : 1.0f);
  }
};

template <typename K>
__device__ __forceinline__ uint32_t digit_of(K k, int shift, uint32_t mask) {
  return (uint32_t)(k >> shift) & mask;
}

// counts[d * tiles + t] = keys of tile t with digit d (d <= mask).
template <typename K, class Src>
__global__ void __launch_bounds__(kSortThreads)
    radix_hist_kernel(Src S, uint64_t n, int shift, uint32_t mask, uint32_t tiles,
                      uint32_t* __restrict__ counts) {
  __shared__ uint32_t h[kRadix];
  for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    for (uint32_t d = threadIdx.x; d <= mask; d += kSortThreads) h[d] = 0u;
    __syncthreads();
    const uint64_t base = (uint64_t)t * kSortTile;
    if (base + kSortTile <= n) {  // block-uniform; the order does not matter here
      K k[kSortItems / 4][4];
#pragma unroll
      for (int i = 0; i < kSortItems / 4; i++)
        S.key4(base + 4 * ((uint64_t)i * kSortThreads + threadIdx.x), k[i]);
#pragma unroll
      for (int i = 0; i < kSortItems; i++)
        atomicAdd(&h[digit_of(k[i / 4][i % 4], shift, mask)], 1u);
    } else {
      for (int i = 0; i < kSortItems; i++) {
        const uint64_t j = base + (uint64_t)i * kSortThreads + threadIdx.x;
        if (j < n) atomicAdd(&h[digit_of(S.key(j), shift, mask)], 1u);
      }
    }
    __syncthreads();
    for (uint32_t d = threadIdx.x; d <= mask; d += kSortThreads)
      counts[(uint64_t)d * tiles + t] = h[d];
    __syncthreads();
  }
}

// Stable scatter of one tile: warp w owns keys [w*256, (w+1)*256) of the
// tile, in order; offsets holds the scanned counts.  Bound by the memory
// system: (key + payload) bytes in and out per entry.  Each key and payload
// word is read once, into registers (the ranking used to read the keys a
// second time), and the shared-memory reorder turns 4-byte scattered stores
// into runs of tile / digits entries.  Equal digits by ballots, 8 steps
// whatever the digits: __match_any_sync takes a step per distinct value.
template <typename K, class Src, int NP>
__global__ void __launch_bounds__(kSortThreads, 3)
    radix_scatter_kernel(Src S, uint64_t n, int shift, uint32_t mask, uint32_t tiles,
                         const uint32_t* __restrict__ offsets, K* __restrict__ keys_out,
                         uint32_t* __restrict__ out0, uint32_t* __restrict__ out1) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  K* k_sm = reinterpret_cast<K*>(smem_raw);
  uint32_t* p_sm = reinterpret_cast<uint32_t*>(smem_raw + sizeof(K) * kSortTile);
  __shared__ uint32_t wbase[kSortWarps][kRadix];
  __shared__ uint32_t gbase[kRadix];  // output offset of a digit minus its place in the tile
  __shared__ uint32_t scan_sm[33];
  static_assert(kRadix <= kSortThreads, "a thread per digit");
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  const int width = 32 - __clz(mask);
  for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    const uint64_t tile0 = (uint64_t)t * kSortTile;
    const uint32_t cnt = n - tile0 < kSortTile ? (uint32_t)(n - tile0) : kSortTile;
    const uint32_t l0 = wid * kWarpKeys + lane;  // this thread's first key in the tile
    K key[kSortItems];
    if (cnt == kSortTile) {  // block-uniform
#pragma unroll
      for (int i = 0; i < kSortItems; i++) key[i] = S.key(tile0 + l0 + i * 32);
    } else {
#pragma unroll
      for (int i = 0; i < kSortItems; i++)
        key[i] = l0 + i * 32 < cnt ? S.key(tile0 + l0 + i * 32) : K(0);
    }
    for (uint32_t d = lane; d <= mask; d += 32) wbase[wid][d] = 0u;
    __syncwarp();
    uint32_t rank[kSortItems];  // place among the warp's keys of the same digit
#pragma unroll
    for (int i = 0; i < kSortItems; i++) {
      const bool valid = l0 + i * 32 < cnt;
      const uint32_t d = digit_of(key[i], shift, mask);
      unsigned peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
      for (int b = 0; b < 8; b++) {
        if (b < width) {  // warp-uniform
          const bool bit = (d >> b) & 1u;
          const unsigned v = __ballot_sync(0xffffffffu, bit);
          peers &= bit ? v : ~v;
        }
      }
      uint32_t before = 0;
      if (valid) before = wbase[wid][d];
      __syncwarp();
      rank[i] = before + __popc(peers & lt);
      if (valid && (peers & lt) == 0u) wbase[wid][d] = before + __popc(peers);
      __syncwarp();
    }
    __syncthreads();
    {  // a thread per digit: the warps' counts in order, then the digits
      const uint32_t d = threadIdx.x;
      uint32_t total = 0;
      if (d <= mask) {
#pragma unroll
        for (int w = 0; w < kSortWarps; w++) {
          const uint32_t c = wbase[w][d];
          wbase[w][d] = total;
          total += c;
        }
      }
      uint32_t all;
      const uint32_t start = block_exclusive_scan<uint32_t>(total, scan_sm, &all);
      if (d <= mask) {
#pragma unroll
        for (int w = 0; w < kSortWarps; w++) wbase[w][d] += start;
        gbase[d] = offsets[(uint64_t)d * tiles + t] - start;
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kSortItems; i++) {
      if (l0 + i * 32 < cnt) {
        rank[i] += wbase[wid][digit_of(key[i], shift, mask)];  // place in the tile
        k_sm[rank[i]] = key[i];
      }
    }
#pragma unroll
    for (int q = 0; q < NP; q++) {
      uint32_t v[kSortItems];
#pragma unroll
      for (int i = 0; i < kSortItems; i++)
        v[i] = l0 + i * 32 < cnt ? S.pay(tile0 + l0 + i * 32, q) : 0u;
#pragma unroll
      for (int i = 0; i < kSortItems; i++)
        if (l0 + i * 32 < cnt) p_sm[q * kSortTile + rank[i]] = v[i];
    }
    __syncthreads();
#pragma unroll 4
    for (uint32_t l = threadIdx.x; l < cnt; l += kSortThreads) {
      const K k = k_sm[l];
      const uint32_t pos = gbase[digit_of(k, shift, mask)] + l;
      keys_out[pos] = k;
      out0[pos] = p_sm[l];
      if (NP > 1) out1[pos] = p_sm[kSortTile + l];
    }
    __syncthreads();
  }
}

unsigned sort_grid(uint32_t tiles) {
  const unsigned cap = sm_count_cached() * 4;  // resident blocks of the passes
  return tiles < cap ? (tiles ? tiles : 1u) : cap;
}

// off[v] = first position whose key is >= v, for v in [0, n]: position j
// writes the rows between the previous key and its own.  Sixteen positions
// per thread, in four 128-bit loads spread over the block (keys is 16-byte
// aligned scratch).
constexpr int kBoundsVecs = 4;
template <typename O>
__global__ void __launch_bounds__(256)
    bounds_from_sorted_kernel(const uint32_t* __restrict__ keys, uint64_t total, uint32_t n,
                              O* __restrict__ off) {
  const uint64_t groups = total / 4 + 1;  // the last one holds position `total`
  const uint64_t stride = (uint64_t)gridDim.x * 256 * kBoundsVecs;
  for (uint64_t b0 = (uint64_t)blockIdx.x * 256 * kBoundsVecs; b0 < groups; b0 += stride) {
    uint32_t k[kBoundsVecs][4], prev[kBoundsVecs];
#pragma unroll
    for (int q = 0; q < kBoundsVecs; q++) {
      const uint64_t g = b0 + q * 256 + threadIdx.x, j0 = 4 * g;
      prev[q] = 0u;
      if (j0 && j0 <= total) prev[q] = keys[j0 - 1] + 1u;  // first row not yet started
      if (j0 + 4 <= total) {
        const uint4 x = reinterpret_cast<const uint4*>(keys)[g];
        k[q][0] = x.x;
        k[q][1] = x.y;
        k[q][2] = x.z;
        k[q][3] = x.w;
      } else {
#pragma unroll
        for (int i = 0; i < 4; i++) k[q][i] = j0 + i < total ? keys[j0 + i] : n;
      }
    }
#pragma unroll
    for (int q = 0; q < kBoundsVecs; q++) {
      const uint64_t j0 = 4 * (b0 + q * 256 + threadIdx.x);
#pragma unroll
      for (int i = 0; i < 4; i++) {
        if (j0 + i > total) break;
        for (uint32_t v = prev[q]; v <= k[q][i] && v <= n; v++) off[v] = (O)(j0 + i);
        prev[q] = k[q][i] + 1u;
      }
    }
  }
}

unsigned bounds_grid(uint64_t total) {
  return (unsigned)std::min<uint64_t>(total / (4 * 256 * kBoundsVecs) + 1, 1u << 16);
}

int bits_for(uint64_t max_key) {
  int b = 0;
  while (b < 64 && (max_key >> b)) b++;
  return b;
}

// Scratch of the sorts below comes from a pool of its own per device, made at
// the first use: with the device's default pool every synchronisation gives
// the freed scratch back to the driver and the next call maps it again (CSR
// of 12 M edges: 6.8 ms a call, 2.0 ms of it kernels).  The pool keeps at
// most kKeepBytes of freed memory, the rest goes back at the stream's next
// synchronisation.  release_sort_scratch() gives all of it back: called when
// an engine of the device ends, when an allocation fails (a sort's here, an
// engine's in its own wrapper) and by lv_release_scratch.  It drops the pool:
// trimming one gives nothing back while the frees queued after a call's wait
// have not been waited for, and a pool must not outlive the device's context.
// Blocks in use stay valid until they are freed.  Allocations are
// stream-ordered, so streams and threads may share the pool.
constexpr uint64_t kKeepBytes = 512ull << 20;
constexpr int kMaxDevices = 64;
std::mutex g_pool_mu;  // held over an allocation: the pool may be dropped
cudaMemPool_t g_pool[kMaxDevices] = {};

cudaError_t pool_alloc(void** p, size_t bytes, int dev, cudaStream_t st) {
  if (dev < 0 || dev >= kMaxDevices) return cudaMallocAsync(p, bytes, st);
  std::lock_guard<std::mutex> lock(g_pool_mu);
  if (!g_pool[dev]) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.handleTypes = cudaMemHandleTypeNone;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    const cudaError_t e = cudaMemPoolCreate(&pool, &props);
    if (e != cudaSuccess) return e;
    uint64_t keep = kKeepBytes;
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    g_pool[dev] = pool;
  }
  return cudaMallocFromPoolAsync(p, bytes, g_pool[dev], st);
}

// A sort's scratch: stream-ordered blocks, freed when it goes out of scope.
struct Scratch {
  cudaStream_t st;
  void* blocks[8];
  int n = 0;
  explicit Scratch(cudaStream_t s) : st(s) {}
  ~Scratch() {
    for (int i = 0; i < n; i++) cudaFreeAsync(blocks[i], st);
  }
  template <typename T>
  cudaError_t get(T** p, size_t count) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const size_t bytes = std::max<size_t>(count, 1) * sizeof(T);
    e = pool_alloc((void**)p, bytes, dev, st);
    if (e == cudaErrorMemoryAllocation) {  // the pool's unused blocks may be in the way
      cudaGetLastError();
      release_sort_scratch(dev);
      e = pool_alloc((void**)p, bytes, dev, st);
    }
    if (e == cudaSuccess) blocks[n++] = *p;
    return e;
  }
};

// Digit passes of a sort on key_bits bits, and the digit of pass p.
struct Digits {
  int passes, width;
  explicit Digits(int key_bits)
      : passes((key_bits + 7) / 8), width(passes ? (key_bits + passes - 1) / passes : 0) {}
  int shift(int p) const { return p * width; }
  uint32_t mask() const { return (1u << width) - 1u; }
};

// One pass: histogram, scan, scatter from S to (keys_out, out0, out1).
template <typename K, class Src, int NP>
cudaError_t radix_pass(const Src& S, uint64_t n, int shift, uint32_t mask, uint32_t* counts,
                       ScanScratch& scan, K* keys_out, uint32_t* out0, uint32_t* out1,
                       cudaStream_t st) {
  constexpr int smem = (int)((sizeof(K) + NP * sizeof(uint32_t)) * kSortTile);
  cudaError_t e = cudaFuncSetAttribute(radix_scatter_kernel<K, Src, NP>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  const uint32_t tiles = (uint32_t)((n + kSortTile - 1) / kSortTile);
  const unsigned grid = sort_grid(tiles);
  (count_launches(1), radix_hist_kernel<K, Src><<<grid, kSortThreads, 0, st>>>(S, n, shift, mask,
                                                                               tiles, counts));
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  e = exclusive_scan_u32(counts, counts, (size_t)tiles * (mask + 1), nullptr, scan, st);
  if (e != cudaSuccess) return e;
  (count_launches(1), radix_scatter_kernel<K, Src, NP><<<grid, kSortThreads, smem, st>>>(
                          S, n, shift, mask, tiles, counts, keys_out, out0, out1));
  return cudaGetLastError();
}

}  // namespace

size_t radix_sort_scratch_words(uint64_t n) {
  const uint64_t tiles = (n + kSortTile - 1) / kSortTile;
  return (size_t)tiles * kRadix + 64;
}

template <typename K>
cudaError_t radix_sort_pairs(K* keys, uint32_t* vals, K* keys_alt, uint32_t* vals_alt,
                             uint64_t n, int key_bits, uint32_t* counts, ScanScratch& S,
                             cudaStream_t st, bool* result_in_alt) {
  *result_in_alt = false;
  if (n <= 1 || key_bits <= 0) return cudaSuccess;
  const Digits D(key_bits);
  for (int p = 0; p < D.passes; p++) {
    ArraySource<K, 1> src{keys, {vals}};
    cudaError_t e = radix_pass<K, ArraySource<K, 1>, 1>(src, n, D.shift(p), D.mask(), counts, S,
                                                        keys_alt, vals_alt, nullptr, st);
    if (e != cudaSuccess) return e;
    std::swap(keys, keys_alt);
    std::swap(vals, vals_alt);
    *result_in_alt = !*result_in_alt;
  }
  return cudaSuccess;
}

template cudaError_t radix_sort_pairs<uint64_t>(uint64_t*, uint32_t*, uint64_t*, uint32_t*,
                                                uint64_t, int, uint32_t*, ScanScratch&,
                                                cudaStream_t, bool*);

void release_sort_scratch(int device) {
  if (device < 0 || device >= kMaxDevices) return;
  std::lock_guard<std::mutex> lock(g_pool_mu);
  if (g_pool[device]) cudaMemPoolDestroy(g_pool[device]);
  g_pool[device] = nullptr;
}

cudaError_t csr_from_edges_device(uint32_t n, uint64_t m, const uint32_t* src,
                                  const uint32_t* dst, const float* w, uint64_t* off,
                                  uint32_t* col, float* wout, uint64_t* nnz_host,
                                  uint32_t* bad_host, cudaStream_t st) {
  const uint64_t total = 2 * m;
  const Digits D(bits_for(n));  // keys 0..n
  // at least one pass: it checks the indices and writes the entries
  const int passes = std::max(1, D.passes);
  uint32_t *keys[2] = {nullptr, nullptr}, *col2 = nullptr, *w2 = nullptr;
  uint32_t *counts = nullptr, *bad = nullptr;
  Scratch tmp(st);
  ScanScratch S;
  unsigned char* scan_buf = nullptr;
  const size_t cw = radix_sort_scratch_words(total);
  S.bytes = scan_scratch_bytes(cw);
  cudaError_t e;
  if ((e = tmp.get(&keys[0], total)) != cudaSuccess) return e;
  if (passes > 1 && ((e = tmp.get(&keys[1], total)) != cudaSuccess ||
                     (e = tmp.get(&col2, total)) != cudaSuccess ||
                     (e = tmp.get(&w2, total)) != cudaSuccess))
    return e;
  if ((e = tmp.get(&counts, cw)) != cudaSuccess || (e = tmp.get(&bad, 1)) != cudaSuccess ||
      (e = tmp.get(&scan_buf, S.bytes)) != cudaSuccess)
    return e;
  S.buf = scan_buf;
  if ((e = cudaMemsetAsync(bad, 0, sizeof(uint32_t), st)) != cudaSuccess) return e;
  // the columns and weights alternate between the scratch and the caller's
  // arrays so that the last pass writes the caller's
  uint32_t* wout_u = reinterpret_cast<uint32_t*>(wout);
  for (int p = 0; total && p < passes; p++) {
    const int left = passes - 1 - p;  // passes after this one
    uint32_t* kd = keys[left & 1];
    uint32_t* cd = (left & 1) ? col2 : col;
    uint32_t* wd = (left & 1) ? w2 : wout_u;
    if (p == 0) {
      const EdgeSource es{src, dst, w, n, bad};
      e = radix_pass<uint32_t, EdgeSource, 2>(es, total, D.shift(0), D.mask(), counts, S, kd, cd,
                                              wd, st);
    } else {
      const ArraySource<uint32_t, 2> as{
          keys[~left & 1], {(left & 1) ? col : col2, (left & 1) ? wout_u : w2}};
      e = radix_pass<uint32_t, ArraySource<uint32_t, 2>, 2>(as, total, D.shift(p), D.mask(),
                                                            counts, S, kd, cd, wd, st);
    }
    if (e != cudaSuccess) return e;
  }
  const unsigned gb = bounds_grid(total);
  (count_launches(1), bounds_from_sorted_kernel<uint64_t><<<gb, 256, 0, st>>>(keys[0], total, n,
                                                                              off));
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  if ((e = cudaMemcpyAsync(nnz_host, off + n, sizeof(uint64_t), cudaMemcpyDeviceToHost, st)) !=
      cudaSuccess)
    return e;
  if ((e = cudaMemcpyAsync(bad_host, bad, sizeof(uint32_t), cudaMemcpyDeviceToHost, st)) !=
      cudaSuccess)
    return e;
  return counted_sync(st);
}

cudaError_t group_by_community(const uint32_t* part, uint32_t n, uint32_t n_comm,
                               uint32_t* out /* [n_comm + 1 + n] */, cudaStream_t st) {
  const Digits D(bits_for(n_comm ? n_comm - 1 : 0));
  uint32_t *keys[2] = {nullptr, nullptr}, *vals2 = nullptr, *counts = nullptr;
  Scratch tmp(st);
  ScanScratch S;
  unsigned char* scan_buf = nullptr;
  const size_t cw = radix_sort_scratch_words(n);
  S.bytes = scan_scratch_bytes(cw);
  cudaError_t e;
  if ((e = tmp.get(&keys[0], n)) != cudaSuccess || (e = tmp.get(&keys[1], n)) != cudaSuccess ||
      (e = tmp.get(&vals2, n)) != cudaSuccess || (e = tmp.get(&counts, cw)) != cudaSuccess ||
      (e = tmp.get(&scan_buf, S.bytes)) != cudaSuccess)
    return e;
  S.buf = scan_buf;
  // vertices start in ascending order and the sort is stable: each
  // community's members come out ascending (utils.cu:280-289 prints them so).
  // At least one pass: with one community it only writes the vertices.
  uint32_t* members = out + n_comm + 1;
  const int passes = std::max(1, D.passes);
  for (int p = 0; n && p < passes; p++) {
    const int left = passes - 1 - p;
    uint32_t* vd = (left & 1) ? vals2 : members;
    if (p == 0) {
      const IndexSource<uint32_t> is{part};
      e = radix_pass<uint32_t, IndexSource<uint32_t>, 1>(is, n, 0, D.mask(), counts, S,
                                                         keys[left & 1], vd, nullptr, st);
    } else {
      const ArraySource<uint32_t, 1> as{keys[~left & 1], {(left & 1) ? members : vals2}};
      e = radix_pass<uint32_t, ArraySource<uint32_t, 1>, 1>(as, n, D.shift(p), D.mask(), counts,
                                                            S, keys[left & 1], vd, nullptr, st);
    }
    if (e != cudaSuccess) return e;
  }
  const unsigned g = bounds_grid(n);
  (count_launches(1), bounds_from_sorted_kernel<uint32_t><<<g, 256, 0, st>>>(keys[0], n, n_comm,
                                                                             out));
  return cudaGetLastError();
}

}  // namespace lvb
