// primitives.cu -- scans, reductions and segmented sorts written for this library
// (no Thrust/CUB on the product path).
#include <map>
#include <mutex>
#include <tuple>

#include "common.cuh"

namespace femgpu {

void ensure_dynamic_smem(const void* func, size_t bytes) {
  static std::mutex mu;
  static std::map<std::pair<int, const void*>, size_t> set;
  int dev = 0;
  FG_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  size_t& cur = set[{dev, func}];
  if (bytes <= cur) return;
  FG_CUDA(cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  cur = bytes;
}


int largest_cluster(const void* func, int threads, int most, size_t smem) {
  static std::mutex mu;
  static std::map<std::tuple<int, const void*, size_t>, int> known;
  int dev = 0;
  FG_CUDA(cudaGetDevice(&dev));
  if (smem > 0) ensure_dynamic_smem(func, smem);
  std::lock_guard<std::mutex> lock(mu);
  int& size = known[std::make_tuple(dev, func, smem)];
  if (size > 0) return size;
  if (most > 8) FG_CUDA(cudaFuncSetAttribute(func, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  for (int c = most; c > 1; c >>= 1) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)c);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)c;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, func, &cfg) == cudaSuccess && clusters > 0) return size = c;
    (void)cudaGetLastError();
  }
  return size = 1;
}

namespace {

#define FG_RUN(...)    \
  do {                 \
    __VA_ARGS__;       \
    FG_CHECK_LAUNCH(); \
  } while (0)

// ---- scans ----------------------------------------------------------------------
// Setup runs about 20 scans per level, most of them over a few thousand counts, where a
// launch (2.2-3 us back to back) costs more than the work: up to kScanOne counts are
// scanned by one block that carries its total from tile to tile and writes the total entry
// itself (one launch; a scan with separate kernels for the saved last entry, the tiles, the
// tile sums, their addition and the total took three to five).  Longer arrays take two
// launches: tile sums, then every block adds up the sums before its tile and scans it.
// 2 k counts: 7.8 -> 3.6 us of device time; 2.1 M: 28 -> 12 us.
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;
constexpr int64_t kScanOne = 2 * kScanTile;   // two tiles by one block: 4.6 us, as two launches
constexpr int64_t kScanSumsInBlock = 2048;    // tile sums that every block adds up by itself

// Block-wide exclusive scan of one value per thread; *total gets the block's sum.
__device__ __forceinline__ int32_t block_exclusive_scan(int32_t v, int32_t* warp_sums, int32_t* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int32_t w = (lane < (int)(blockDim.x >> 5)) ? warp_sums[lane] : 0;
    int32_t ws = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int32_t y = __shfl_up_sync(0xffffffffu, ws, o);
      if (lane >= o) ws += y;
    }
    warp_sums[lane] = ws - w;  // exclusive warp offsets
    if (lane == 31) *total = ws;
  }
  __syncthreads();
  return warp_sums[warp] + x - v;
}

// A thread's kScanItems consecutive values of a tile (zero past n): two 16-byte loads when
// the array and the range allow it.
__device__ __forceinline__ void scan_load(const int32_t* in, int64_t base, int64_t n, int32_t v[kScanItems]) {
  if (base + kScanItems <= n && (reinterpret_cast<uintptr_t>(in) & 15) == 0) {
    const int4* p = reinterpret_cast<const int4*>(in + base);
    const int4 a = p[0], b = p[1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    return;
  }
#pragma unroll
  for (int k = 0; k < kScanItems; k++) v[k] = base + k < n ? in[base + k] : 0;
}

// Scans tile `tile` from `carry`; returns the tile's sum.  The block reads its tile before
// it writes it, so in and out may be the same array.
template <bool INCLUSIVE>
__device__ __forceinline__ int32_t scan_tile(const int32_t* in, int32_t* out, int64_t n, int64_t tile, int32_t carry,
                                             int32_t* warp_sums, int32_t* total) {
  const int64_t base = tile * kScanTile + (int64_t)threadIdx.x * kScanItems;
  int32_t v[kScanItems];
  scan_load(in, base, n, v);
  int32_t local = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; k++) local += v[k];
  int32_t off = carry + block_exclusive_scan(local, warp_sums, total);
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    const int32_t e = off;
    off += v[k];
    v[k] = INCLUSIVE ? off : e;
  }
  if (base + kScanItems <= n && (reinterpret_cast<uintptr_t>(out) & 15) == 0) {
    int4* p = reinterpret_cast<int4*>(out + base);
    p[0] = make_int4(v[0], v[1], v[2], v[3]);
    p[1] = make_int4(v[4], v[5], v[6], v[7]);
  } else {
#pragma unroll
    for (int k = 0; k < kScanItems; k++)
      if (base + k < n) out[base + k] = v[k];
  }
  return *total;
}

template <bool INCLUSIVE>
__global__ void __launch_bounds__(kScanThreads) scan_one_kernel(const int32_t* in, int32_t* out, int64_t n) {
  __shared__ int32_t warp_sums[32];
  __shared__ int32_t total;
  int32_t carry = 0;
  for (int64_t t = 0; t * kScanTile < n; t++) {
    carry += scan_tile<INCLUSIVE>(in, out, n, t, carry, warp_sums, &total);
    __syncthreads();  // warp_sums and total are free for the next tile
  }
  if (!INCLUSIVE && threadIdx.x == 0) out[n] = carry;
}

__global__ void __launch_bounds__(kScanThreads) tile_sums_kernel(const int32_t* in, int64_t n, int32_t* sums) {
  __shared__ int32_t ws[32];
  int32_t v[kScanItems], s = 0;
  scan_load(in, (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems, n, v);
#pragma unroll
  for (int k = 0; k < kScanItems; k++) s += v[k];
  s = __reduce_add_sync(0xffffffffu, s);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = __reduce_add_sync(0xffffffffu, ws[threadIdx.x]);
    if (threadIdx.x == 0) sums[blockIdx.x] = s;
  }
}

// `scanned`: sums holds the exclusive scan of the tile sums, else the sums themselves.
template <bool INCLUSIVE>
__global__ void __launch_bounds__(kScanThreads) scan_tiles_kernel(const int32_t* in, int32_t* out, int64_t n,
                                                                  const int32_t* sums, int scanned) {
  __shared__ int32_t warp_sums[32];
  __shared__ int32_t total;
  int32_t carry;
  if (scanned) {
    carry = sums[blockIdx.x];
  } else {
    int32_t s = 0;
    for (int t = threadIdx.x; t < (int)blockIdx.x; t += kScanThreads) s += sums[t];
    block_exclusive_scan(s, warp_sums, &total);
    carry = total;
    __syncthreads();
  }
  carry += scan_tile<INCLUSIVE>(in, out, n, blockIdx.x, carry, warp_sums, &total);
  if (!INCLUSIVE && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) out[n] = carry;
}

template <bool INCLUSIVE>
void scan(const int32_t* in, int32_t* out, int64_t n, cudaStream_t s) {
  if (n <= kScanOne) {
    if (INCLUSIVE && n <= 0) return;
    FG_RUN(scan_one_kernel<INCLUSIVE><<<1, kScanThreads, 0, s>>>(in, out, n < 0 ? 0 : n));
    return;
  }
  const int64_t tiles = (n + kScanTile - 1) / kScanTile;
  DBuf<int32_t> sums(tiles + 1, s);
  FG_RUN(tile_sums_kernel<<<(unsigned)tiles, kScanThreads, 0, s>>>(in, n, sums.p));
  const bool deep = tiles > kScanSumsInBlock;
  if (deep) scan<false>(sums.p, sums.p, tiles, s);
  FG_RUN(scan_tiles_kernel<INCLUSIVE><<<(unsigned)tiles, kScanThreads, 0, s>>>(in, out, n, sums.p, deep));
}

// One block: the maximum of a[0 .. n) straight to *out.
__global__ void __launch_bounds__(1024) reduce_max_one_kernel(const int32_t* a, int64_t n, int32_t* out) {
  __shared__ int32_t wm[32];
  int32_t m = INT32_MIN;
#pragma unroll 4
  for (int64_t i = threadIdx.x; i < n; i += 1024) m = max(m, a[i]);
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 32) {
    m = __reduce_max_sync(0xffffffffu, wm[threadIdx.x]);
    if (threadIdx.x == 0) *out = m;
  }
}

__global__ void reduce_max_kernel(const int32_t* a, int64_t n, int32_t* out) {
  int32_t m = INT32_MIN;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    m = max(m, a[i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  // one atomic per block
  __shared__ int32_t wm[32];
  if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 32) {
    m = threadIdx.x < (blockDim.x >> 5) ? wm[threadIdx.x] : INT32_MIN;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (threadIdx.x == 0) atomicMax(out, m);
  }
}

__global__ void count_equal_kernel(const int32_t* a, int64_t n, int32_t v, unsigned long long* out) {
  unsigned c = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    c += (a[i] == v);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  // one atomic per block
  __shared__ unsigned wc[32];
  if ((threadIdx.x & 31) == 0) wc[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x < 32) {
    c = threadIdx.x < (blockDim.x >> 5) ? wc[threadIdx.x] : 0u;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if (threadIdx.x == 0 && c) atomicAdd(out, (unsigned long long)c);
  }
}

__global__ void fill_kernel(int32_t* a, int64_t n, int32_t v) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) a[i] = v;
}
__global__ void iota_kernel(int32_t* a, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    a[i] = (int32_t)i;
}

int reduce_grid(int64_t n) {
  int64_t g = (n + 255) / 256;
  return (int)(g < 1 ? 1 : (g > 152 * 16 ? 152 * 16 : g));
}

// ---- segmented sort ----------------------------------------------------------
constexpr int kWarpCap = 1024;   // per-warp shared-memory capacity (ints)
constexpr int kWarpsPerBlock = 4;
constexpr int kBlockCap = 8192;  // per-block capacity (ints)

// Compacts the sorted run s[0..len) to its unique values at dst; returns count.
template <class Sync>
__device__ int unique_write(const int32_t* s, int len, int32_t* dst, int tid, int nthr, int32_t* scratch_count,
                            Sync sync) {
  // sequential-by-chunk ballot compaction works only inside one warp; blocks use
  // a simple two-step approach on the scratch counter.
  int count = 0;
  if (nthr == 32) {
    for (int base = 0; base < len; base += 32) {
      int p = base + tid;
      bool keep = p < len && (p == 0 || s[p] != s[p - 1]);
      unsigned m = __ballot_sync(0xffffffffu, keep);
      if (keep) dst[count + __popc(m & ((1u << tid) - 1u))] = s[p];
      count += __popc(m);
    }
    return count;
  }
  // block: one thread writes (blocks are only used for rare long segments)
  if (tid == 0) {
    int c = 0;
    for (int p = 0; p < len; p++)
      if (p == 0 || s[p] != s[p - 1]) dst[c++] = s[p];
    *scratch_count = c;
  }
  sync();
  return *scratch_count;
}

__global__ void segsort_warp_kernel(int32_t* vals, const int32_t* off, int nseg, int32_t* ucount) {
  __shared__ int32_t sm[kWarpsPerBlock][kWarpCap];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int seg = blockIdx.x * kWarpsPerBlock + w;
  if (seg >= nseg) return;
  int b = off[seg], e = off[seg + 1], len = e - b;
  if (len > kWarpCap) return;
  int32_t* s = sm[w];
  int np2 = next_pow2(len < 2 ? 2 : len);
  for (int i = lane; i < np2; i += 32) s[i] = (i < len) ? vals[b + i] : INT32_MAX;
  __syncwarp();
  bitonic_sort_shared(s, np2, lane, 32, WarpSync());
  if (ucount) {
    int c = unique_write(s, len, vals + b, lane, 32, nullptr, WarpSync());
    if (lane == 0) ucount[seg] = c;
  } else {
    for (int i = lane; i < len; i += 32) vals[b + i] = s[i];
  }
}

// Heap sort in global memory for segments beyond the shared-memory tiers.
__device__ void sift_down(int32_t* a, int start, int end) {
  int root = start;
  while (2 * root + 1 <= end) {
    int child = 2 * root + 1, sw = root;
    if (a[sw] < a[child]) sw = child;
    if (child + 1 <= end && a[sw] < a[child + 1]) sw = child + 1;
    if (sw == root) return;
    int32_t t = a[root];
    a[root] = a[sw];
    a[sw] = t;
    root = sw;
  }
}

// Segments longer than a warp's capacity: block b looks at segments b, b + grid, b + 2 grid, ...
// (1024 at a time), lists the long ones and sorts them one after the other, so the host needs
// no look at the lengths.  Lists of that length are rare (a vertex in more than 256 elements);
// without one the kernel reads the offsets and ends (4 us for a million).  Neighbouring segments
// go to different blocks, because vertices of many elements are often numbered together: 1000
// vertices of 400 triangles each, set_mesh 33.6 -> 1.25 ms; 200 of 3000 triangles, 1577 -> 12 ms.
__global__ void __launch_bounds__(1024) segsort_long_kernel(int32_t* vals, const int32_t* off, int nseg,
                                                            int32_t* ucount) {
  __shared__ int32_t s[kBlockCap];
  __shared__ int32_t list[1024];
  __shared__ int32_t cnt, nlist;
  for (int64_t s0 = blockIdx.x; s0 < nseg; s0 += (int64_t)gridDim.x * 1024) {
    const int64_t mine = s0 + (int64_t)gridDim.x * threadIdx.x;
    const bool is_long = mine < nseg && off[mine + 1] - off[mine] > kWarpCap;
    if (!__syncthreads_or(is_long)) continue;
    if (threadIdx.x == 0) nlist = 0;
    __syncthreads();
    if (is_long) list[atomicAdd(&nlist, 1)] = (int)mine;
    __syncthreads();
    for (int k = 0; k < nlist; k++) {
      const int seg = list[k], b = off[seg], len = off[seg + 1] - b;
      if (len <= kBlockCap) {
        const int np2 = next_pow2(len);
        for (int i = threadIdx.x; i < np2; i += blockDim.x) s[i] = (i < len) ? vals[b + i] : INT32_MAX;
        __syncthreads();
        bitonic_sort_shared(s, np2, threadIdx.x, blockDim.x, BlockSync());
        if (ucount) {
          const int c = unique_write(s, len, vals + b, threadIdx.x, blockDim.x, &cnt, BlockSync());
          if (threadIdx.x == 0) ucount[seg] = c;
        } else {
          for (int i = threadIdx.x; i < len; i += blockDim.x) vals[b + i] = s[i];
        }
      } else if (threadIdx.x == 0) {
        int32_t* a = vals + b;
        for (int st = (len - 2) / 2; st >= 0; st--) sift_down(a, st, len - 1);
        for (int end = len - 1; end > 0; end--) {
          const int32_t t = a[0];
          a[0] = a[end];
          a[end] = t;
          sift_down(a, 0, end - 1);
        }
        if (ucount) {
          int c = 0;
          for (int p = 0; p < len; p++)
            if (p == 0 || a[p] != a[p - 1]) a[c++] = a[p];
          ucount[seg] = c;
        }
      }
      __syncthreads();
    }
    __syncthreads();
  }
}

}  // namespace

void exclusive_scan_async(const int32_t* in, int32_t* out, int64_t n, cudaStream_t s) { scan<false>(in, out, n, s); }

int64_t exclusive_scan(const int32_t* in, int32_t* out, int64_t n, cudaStream_t s) {
  exclusive_scan_async(in, out, n, s);
  return (int64_t)read_scalar(out + n, s);
}

void inclusive_scan(const int32_t* in, int32_t* out, int64_t n, cudaStream_t s) { scan<true>(in, out, n, s); }

void reduce_max_async(const int32_t* a, int64_t n, int32_t* out, cudaStream_t s) {
  if (n <= kScanOne) {
    FG_RUN(reduce_max_one_kernel<<<1, 1024, 0, s>>>(a, n, out));
    return;
  }
  fill_i32(out, 1, INT32_MIN, s);
  FG_RUN(reduce_max_kernel<<<reduce_grid(n), 256, 0, s>>>(a, n, out));
}

int32_t reduce_max(const int32_t* a, int64_t n, cudaStream_t s) {
  DBuf<int32_t> out(1, s);
  reduce_max_async(a, n, out.p, s);
  return read_scalar(out.p, s);
}

int64_t count_equal(const int32_t* a, int64_t n, int32_t value, cudaStream_t s) {
  DBuf<unsigned long long> out(1, s);
  out.zero();
  if (n > 0) {
    count_equal_kernel<<<reduce_grid(n), 256, 0, s>>>(a, n, value, out.p);
    FG_CHECK_LAUNCH();
  }
  return (int64_t)read_scalar(out.p, s);
}

void fill_i32(int32_t* a, int64_t n, int32_t v, cudaStream_t s) {
  if (n <= 0) return;
  fill_kernel<<<reduce_grid(n), 256, 0, s>>>(a, n, v);
  FG_CHECK_LAUNCH();
}

void iota_i32(int32_t* a, int64_t n, cudaStream_t s) {
  if (n <= 0) return;
  iota_kernel<<<reduce_grid(n), 256, 0, s>>>(a, n);
  FG_CHECK_LAUNCH();
}

void segmented_sort_i32(int32_t* vals, const int32_t* off, int nseg, int32_t* ucount, cudaStream_t s) {
  if (nseg <= 0) return;
  FG_RUN(segsort_warp_kernel<<<grid_for(nseg, kWarpsPerBlock), 32 * kWarpsPerBlock, 0, s>>>(vals, off, nseg, ucount));
  FG_RUN(segsort_long_kernel<<<nseg < 152 * 2 ? nseg : 152 * 2, 1024, 0, s>>>(vals, off, nseg, ucount));
}

}  // namespace femgpu
