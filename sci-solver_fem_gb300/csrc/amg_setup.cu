// amg_setup.cu -- smoothed-aggregation hierarchy built on the device.
//
// Per level (AMG::setup, src/core/cuda/amg.cu:80-144; createNextLevel,
// smoothedMG_amg_level.cu:403-494):
//   1. OldMIS two-level aggregation of the level graph (ComputePermutationMethods.cu:22-151):
//      seeded distance-2 randomized MIS -> aggregates (min size 9) -> distance-1 MIS on
//      the aggregate graph -> partitions of <= partitionMaxSize rows;
//   2. the permutation that makes aggregates and partitions contiguous;
//   3. Ap = perm(A), the in/out-of-partition split used by the smoother;
//   4. P = (I - omega D^-1 Ap) T, R = P^T;
//   5. A_next = R (Ap P), each product row accumulated in generation order by the
//      tier its size calls for: a per-thread column list (large levels), a warp hash
//      table, a block hash table or a dense accumulator;
//   6. each parent's R rows and P columns put in the child's order, and the FP64 outer
//      operator in level-0 order as 32-row slices.
// Integer results are bit-identical to the CPU oracle for the same seed; floating
// results use fixed summation orders (generation order, ascending column), so they are
// too.
#include <algorithm>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cmath>
#include <limits>
#include <type_traits>
#include <vector>

#include <cooperative_groups.h>

#include "context.cuh"

namespace cg = cooperative_groups;

namespace femgpu {

namespace {

constexpr int kCap = 100000;  // bound on every data-dependent loop (error, never spin)

// Setup phase timer (FEMGPU_PROFILE): stream-synchronised wall time per phase with
// the kernel launches and host reads it took.
struct PhaseTimer {
  bool on;
  cudaStream_t s;
  int level;
  std::chrono::steady_clock::time_point t0;
  int64_t syncs0 = 0, launches0 = 0;
  PhaseTimer(cudaStream_t st, int lvl) : on(getenv("FEMGPU_PROFILE") != nullptr), s(st), level(lvl) {
    if (on) {
      cudaStreamSynchronize(s);
      t0 = std::chrono::steady_clock::now();
      syncs0 = g_host_syncs.load();
      launches0 = g_kernel_launches.load();
    }
  }
  void mark(const char* what) {
    if (!on) return;
    cudaStreamSynchronize(s);
    auto t = std::chrono::steady_clock::now();
    const int64_t sy = g_host_syncs.load(), la = g_kernel_launches.load();
    fprintf(stderr, "[femgpu setup] level %d %-10s %8.3f ms  %5lld launches %4lld host reads\n", level, what,
            std::chrono::duration<double, std::milli>(t - t0).count(), (long long)(la - launches0),
            (long long)(sy - syncs0));
    t0 = t;
    syncs0 = sy;
    launches0 = la;
  }
};

// ---------------------------------------------------------------------------------
// glibc rand() stream (TYPE_3 additive feedback generator), host side: the
// reference draws 32768 seeds with rand() after srand() (randomizedMIS_GPU.cu:195-201).
void glibc_rand_stream(uint32_t seed, int count, std::vector<uint32_t>& out) {
  std::vector<uint32_t> st(344 + (size_t)count);
  int32_t s0 = (int32_t)(seed ? seed : 1u);
  st[0] = (uint32_t)s0;
  int64_t w = s0;
  for (int i = 1; i < 31; i++) {
    w = (16807LL * w) % 2147483647LL;
    if (w < 0) w += 2147483647LL;
    st[i] = (uint32_t)w;
  }
  for (int i = 31; i < 34; i++) st[i] = st[i - 31];
  for (size_t i = 34; i < st.size(); i++) st[i] = st[i - 31] + st[i - 3];
  out.resize(count);
  for (int k = 0; k < count; k++) out[k] = st[344 + (size_t)k] >> 1;
}

__device__ __forceinline__ uint32_t taus(uint32_t z) {
  uint32_t b = (((z << 13) ^ z) >> 19);
  return (z << 12) ^ b;
}

// ---- randomized MIS (randomizedMIS_GPU.cu:3-152) ---------------------------------
__global__ void mis_randoms_kernel(int n, int iterations, uint32_t* randoms, const uint32_t* __restrict__ seeds) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 32768) return;
  uint32_t z = seeds[t];
  int off = t;
  for (int i = 0; i < iterations; i++)
    if (off < n) {
      z = taus(z);
      randoms[off] = z;
      off += 32768;
    }
}

// A node's (value, origin) pair packed as value << 32 | origin: the reference's update
// (take a neighbour with a larger value, or the same positive value and a larger
// origin) is the maximum of the packed keys over the node and its neighbours with a
// positive value.
__device__ __forceinline__ uint64_t mis_key(int32_t best, int32_t origin) {
  return ((uint64_t)(uint32_t)best << 32) | (uint32_t)origin;
}

__global__ void mis_first_init_kernel(int n, const uint32_t* randoms, uint64_t* key) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) key[i] = mis_key((int32_t)(randoms[i] % 1000000u), i);
}

__global__ void mis_init_kernel(int n, uint32_t* randoms, uint64_t* key, const int32_t* mis) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    uint32_t z = taus(randoms[i]);
    int st = mis[i];
    key[i] = mis_key(st == -1 ? (int32_t)(z % 1000000u) : (st == 1 ? 1000001 : 0), i);
    randoms[i] = z;
  }
}

__global__ void mis_iterate_kernel(int n, const uint64_t* __restrict__ kin, uint64_t* __restrict__ kout,
                                   const int32_t* __restrict__ xadj, const int32_t* __restrict__ adj, int32_t* mis,
                                   int32_t* incomplete, int final_pass) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint64_t k = kin[i];
  if ((k >> 32) < 1000001u) {
    // neighbours in groups of 8: all indices, then all keys, so the loads overlap
    const int e1 = xadj[i + 1];
    for (int e0 = xadj[i]; e0 < e1; e0 += 8) {
      int nb[8];
      uint64_t kn[8];
#pragma unroll
      for (int q = 0; q < 8; q++) nb[q] = e0 + q < e1 ? adj[e0 + q] : i;
#pragma unroll
      for (int q = 0; q < 8; q++) kn[q] = kin[nb[q]];
#pragma unroll
      for (int q = 0; q < 8; q++)
        if ((kn[q] >> 32) > 0u && kn[q] > k) k = kn[q];
    }
  }
  kout[i] = k;
  if (final_pass) {
    const int best = (int)(k >> 32), org = (int)(uint32_t)k;
    int st = -1;
    if (org == i) st = 1;
    else if (best == 1000001) st = 0;
    mis[i] = st;
    // one store per warp with an undecided node (a single flag address)
    const unsigned undecided = __ballot_sync(__activemask(), st == -1);
    if (undecided && (threadIdx.x & 31) == (__ffs(__activemask()) - 1)) *incomplete = 1;
  }
}

// The 32768 generator seeds of cfg.seed, made once per handle and seed.
const uint32_t* mis_seeds(Ctx& c) {
  if (c.mis_seeds.n == 0 || c.mis_seeds_of != c.cfg.seed) {
    std::vector<uint32_t> seeds;
    glibc_rand_stream(c.cfg.seed, 32768, seeds);
    c.mis_seeds.alloc(32768, c.stream);
    c.mis_seeds.upload(seeds.data(), 32768);
    FG_CUDA(cudaStreamSynchronize(c.stream));  // the host copy ends here
    c.mis_seeds_of = c.cfg.seed;
  }
  return c.mis_seeds.p;
}

void random_mis(Ctx& c, int n, const int32_t* xadj, const int32_t* adj, int k, DBuf<int32_t>& mis) {
  cudaStream_t s = c.stream;
  PhaseTimer pt(s, -5);
  mis.alloc(n, s);
  fill_i32(mis.p, n, -1, s);
  const uint32_t* seeds = mis_seeds(c);
  DBuf<uint32_t> randoms(n, s);
  DBuf<uint64_t> k0(n, s), k1(n, s);
  DBuf<int32_t> flag(1, s);
  FG_LAUNCH(mis_randoms_kernel, 128, 256, 0, s, n, (n + 32767) / 32768, randoms.p, seeds);
  FG_LAUNCH(mis_first_init_kernel, grid_for(n, 256), 256, 0, s, n, randoms.p, k0.p);
  pt.mark("mis init");
  // Rounds are enqueued in batches and the flag of a batch's last round is read once: a
  // round after the one that completes the set changes nothing (decided nodes keep their
  // state), so the extra rounds only cost time.  Small levels, where a host
  // round trip costs more than a round, take larger batches.
  const int batch = n < (1 << 18) ? 4 : 2;
  for (int round = 0;; round++) {
    FG_REQUIRE(round < kCap, FEMGPU_ERR_LIMIT, "randomized MIS did not complete");
    if (round > 0) FG_LAUNCH(mis_init_kernel, grid_for(n, 256), 256, 0, s, n, randoms.p, k0.p, mis.p);
    flag.zero();
    uint64_t *ki = k0.p, *ko = k1.p;
    for (int it = 0; it < k; it++) {
      FG_LAUNCH(mis_iterate_kernel, grid_for(n, 256), 256, 0, s, n, ki, ko, xadj, adj, mis.p, flag.p, it == k - 1);
      std::swap(ki, ko);
    }
    if (ki != k0.p) std::swap(k0, k1);  // keep k0 as the next round's input
    if ((round + 1) % batch != 0) continue;
    if (read_scalar(flag.p, s) == 0) break;
    pt.mark("mis rounds");
  }
}

// ---- aggregation helpers (misHelpers.cu) ----------------------------------------------
__global__ void label_roots_kernel(int n, const int32_t* mis, const int32_t* incl, int32_t* part, int32_t* aggregated) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    aggregated[i] = mis[i];
    part[i] = mis[i] == 0 ? -1 : incl[i] - 1;  // ifLabelOne
  }
}

// allocateNodesKernel (misHelpers.cu:13-75): its candidate loop fills every free slot
// with the first aggregated neighbour seen and can never out-count it, so an
// unaggregated node joins the aggregate of its first aggregated neighbour in
// adjacency order.  Writes the full partOut so the buffers can be swapped.
__global__ void allocate_kernel(int n, const int32_t* __restrict__ xadj, const int32_t* __restrict__ adj,
                                const int32_t* __restrict__ pin, int32_t* __restrict__ pout, int32_t* aggregated,
                                int32_t* counters /* [0] unallocated after, [1] changed */) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  bool changed = false, left = false;
  if (i < n) {
    int p = pin[i];
    if (aggregated[i] == 0) {
      int add = -1;
      // first aggregated neighbour in adjacency order, neighbours loaded 8 at a time
      const int e1 = xadj[i + 1];
      for (int e0 = xadj[i]; e0 < e1 && add == -1; e0 += 8) {
        int nb[8], cnd[8];
#pragma unroll
        for (int q = 0; q < 8; q++) nb[q] = e0 + q < e1 ? adj[e0 + q] : -1;
#pragma unroll
        for (int q = 0; q < 8; q++) cnd[q] = nb[q] >= 0 ? pin[nb[q]] : -1;
#pragma unroll
        for (int q = 0; q < 8; q++)
          if (add == -1 && cnd[q] != -1) add = cnd[q];
      }
      p = add;
      if (add != -1) {
        aggregated[i] = 1;
        changed = true;
      } else {
        left = true;
      }
    }
    pout[i] = p;
  }
  // one atomic per block instead of one per node (a single counter address)
  const int nleft = __syncthreads_count(left);
  const int nchanged = __syncthreads_or(changed);
  if (threadIdx.x == 0) {
    if (nleft) atomicAdd(&counters[0], nleft);
    if (nchanged) atomicExch(&counters[1], 1);
  }
}

__global__ void histogram_kernel(int n, const int32_t* part, const int32_t* w, int32_t* sizes) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    int p = part[i];
    if (p >= 0) atomicAdd(&sizes[p], w ? w[i] : 1);
  }
}

__global__ void less_than_kernel(int np, const int32_t* sizes, int threshold, int32_t* flags) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < np) flags[p] = sizes[p] < threshold ? 1 : 0;
}

__global__ void remove_parts_kernel(int n, int32_t* part, const int32_t* rm, const int32_t* sub, int32_t* aggregated) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    int p = part[i];
    int q = rm[p] ? -1 : p - sub[p];
    part[i] = q;
    aggregated[i] = q == -1 ? 0 : 1;
  }
}

// findDesirabilityKernel (misHelpers.cu:297-382) with IEEE float steps spelled out: the
// partition node idx would move to, and the packed (desirability, node) key of the move.
// L2: part and sizes are written by other CTAs of the running kernel (read past L1).
template <bool L2>
__device__ __forceinline__ unsigned long long desirability(int idx, int opt, const int32_t* __restrict__ xadj,
                                                           const int32_t* __restrict__ adj, const int32_t* part,
                                                           const int32_t* sizes, const int32_t* __restrict__ w,
                                                           int& cur, int& addTo) {
  auto ld = [](const int32_t* p) { return L2 ? __ldcg(p) : *p; };
  cur = ld(part + idx);
  int cs = ld(sizes + cur);
  int nw = w[idx];
  int selfAdj = 0;
  addTo = -1;
  float bestD = 0.0f;
  float cwf = __fdiv_rn((float)abs(cs - opt), (float)opt);
  float selfImp = __fmul_rn((float)(abs(cs - opt) - abs((cs - nw) - opt)), cwf);
  if (selfImp > 0) {
    int cand[10], cnt[10];
#pragma unroll
    for (int q = 0; q < 10; q++) {
      cand[q] = -1;
      cnt[q] = 0;
    }
    // neighbours in groups of 8: all indices, then all parts, so the loads overlap
    const int e1 = xadj[idx + 1];
    for (int e0 = xadj[idx]; e0 < e1; e0 += 8) {
      int nb[8], pc[8];
#pragma unroll
      for (int u = 0; u < 8; u++) nb[u] = e0 + u < e1 ? adj[e0 + u] : idx;
#pragma unroll
      for (int u = 0; u < 8; u++) pc[u] = e0 + u < e1 ? ld(part + nb[u]) : -1;
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const int cc = pc[u];
        if (cc == -1) continue;  // past the list's end (every node has a part)
        if (cc == cur) {
          selfAdj++;
          continue;
        }
        // distinct candidates in first-seen order, at most 10 (junk counts of free
        // slots in the reference never reach a used slot)
        bool placed = false;
#pragma unroll
        for (int q = 0; q < 10; q++) {
          const bool here = !placed && (cand[q] == cc || cand[q] == -1);
          cnt[q] += here;
          if (here) cand[q] = cc;
          placed |= here;
        }
      }
    }
    // the reference scans candidates 1..9 (its loop starts at 1)
#pragma unroll
    for (int q = 1; q < 10; q++) {
      if (cand[q] == -1) continue;
      int np_ = cand[q];
      int nsz = ld(sizes + np_);
      float nwf = __fdiv_rn((float)abs(nsz - opt), (float)opt);
      float imp = __fmul_rn((float)(abs(nsz - opt) - abs((nsz + nw) - opt)), nwf);
      imp = __fadd_rn(imp, selfImp);
      float ratio = __fdiv_rn((float)cnt[q], (float)selfAdj);
      imp = __fmul_rn(imp, ratio);
      if (imp > bestD) {
        addTo = np_;
        bestD = imp;
      }
    }
  }
  return ((unsigned long long)__float_as_uint(bestD) << 32) | (unsigned)idx;
}

__global__ void desirability_kernel(int n, int opt, const int32_t* __restrict__ xadj, const int32_t* __restrict__ adj,
                                    const int32_t* __restrict__ part, const int32_t* __restrict__ sizes,
                                    const int32_t* __restrict__ w, int32_t* to,
                                    unsigned long long* best /* per partition: (desirability bits, node) */) {
  int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n) return;
  int cur, add;
  const unsigned long long key = desirability<false>(idx, opt, xadj, adj, part, sizes, w, cur, add);
  to[idx] = add;
  atomicMax(&best[cur], key);
}

// makeSwapsKernel (misHelpers.cu:384-412): per source partition, the node with the
// largest (desirability, index) moves when its desirability exceeds 0.1.
__global__ void swap_kernel(int np, unsigned long long* best, int32_t* part, const int32_t* to, const int32_t* w,
                            int32_t* sizes) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= np) return;
  unsigned long long key = best[p];
  best[p] = 0ull;
  float d = __uint_as_float((unsigned)(key >> 32));
  int idx = (int)(key & 0xffffffffu);
  if ((double)d > .1) {
    int t = to[idx];
    part[idx] = t;
    atomicAdd(&sizes[t], w[idx]);
    atomicAdd(&sizes[p], -w[idx]);
  }
}

// removeRuntyParts / removeRuntyPartitions (misHelpers.cu:744-820).  Returns the
// number of removed parts.  np: the number of parts (labels 0 .. np-1, none empty)
// when the caller tracks it, else -1 (then it is read from the labels).
int remove_small_parts(Ctx& c, int n, DBuf<int32_t>& part, const int32_t* weights, int threshold_mode, int min_size,
                       int full_size, DBuf<int32_t>& aggregated, int np = -1) {
  cudaStream_t s = c.stream;
  if (np < 0) np = reduce_max(part.p, n, s) + 1;
  DBuf<int32_t> sizes(np, s), rm(np + 1, s), sub(np + 1, s);
  sizes.zero();
  FG_LAUNCH(histogram_kernel, grid_for(n, 256), 256, 0, s, n, part.p, weights, sizes.p);
  int threshold = min_size;
  if (threshold_mode == 1) {
    double avg = (double)full_size / np;
    threshold = (int)(avg * .7);
  }
  FG_LAUNCH(less_than_kernel, grid_for(np, 256), 256, 0, s, np, sizes.p, threshold, rm.p);
  int64_t removed = exclusive_scan(rm.p, sub.p, np, s);
  if (removed == 0 && threshold_mode == 0) return 0;
  // subtractions = inclusive scan of the removal flags = exclusive scan shifted by one
  FG_LAUNCH(remove_parts_kernel, grid_for(n, 256), 256, 0, s, n, part.p, rm.p, sub.p + 1, aggregated.p);
  return (int)removed;
}

// np: the number of partitions (labels 0 .. np-1, none empty) when the caller tracks it,
// else -1 (then it is read from the labels).
int restrict_partitions(Ctx& c, int max_size, int full_size, int n, const int32_t* xadj, const int32_t* adj,
                        DBuf<int32_t>& part, const int32_t* w, int np = -1) {
  cudaStream_t s = c.stream;
  if (np < 0) np = reduce_max(part.p, n, s) + 1;
  DBuf<int32_t> sizes(np, s), to(n, s);
  sizes.zero();
  FG_LAUNCH(histogram_kernel, grid_for(n, 256), 256, 0, s, n, part.p, w, sizes.p);
  int avg = full_size / np;
  DBuf<unsigned long long> best(np, s);
  best.zero();
  int largest = reduce_max(sizes.p, np, s);
  int loops = 0;
  while (largest > max_size) {
    FG_REQUIRE(++loops < kCap, FEMGPU_ERR_LIMIT, "partition size restriction did not converge");
    FG_LAUNCH(desirability_kernel, grid_for(n, 256), 256, 0, s, n, avg, xadj, adj, part.p, sizes.p, w, to.p, best.p);
    FG_LAUNCH(swap_kernel, grid_for(np, 256), 256, 0, s, np, best.p, part.p, to.p, w, sizes.p);
    largest = reduce_max(sizes.p, np, s);
  }
  return np;
}

[[noreturn]] void throw_stalled() {
  throw Error(FEMGPU_ERR_LIMIT,
              "aggregation stalled: nodes unreachable from any aggregate, or every aggregate was removed "
              "as undersized");
}

// ---- aggregation of small graphs in one kernel ------------------------------------------
// The whole of aggregate() below (MIS rounds, labels, allocation passes, removal of small
// parts, partition restriction) for a graph of at most kClusterAggEdges edges, as one
// thread-block cluster: CTA c owns a contiguous range of the nodes (and of the parts), the
// arrays stay in L2, and what ended a launch or a read by the host is a cluster barrier
// (0.3 us).  As separate launches these graphs are bound by launches (2.5-4 us each, 25-60 of
// them) and by the flags the host reads (12-20 us each, 5-10 of them).  Every step computes
// what its kernel computes, so the labels are the same.
// The line is drawn by edges, whose gathers the cluster's 16 SMs must do alone (ms per call,
// launches against cluster): 1,590 nodes 0.33 / 0.14; 39,304 nodes with 0.53 M edges 0.49 /
// 0.42; 90,601 nodes with 0.54 M edges 0.60 / 0.30; 80,338 nodes with 1.2 M edges 0.49 / 0.77;
// 132,651 nodes with 1.8 M edges 0.60 / 1.30.
constexpr int kAggThreads = 1024;
constexpr int kAggCtas = 16;  // largest cluster (8 where 16 cannot be scheduled)
constexpr int64_t kClusterAggEdges = 600000;

enum AggStatus { AGG_OK = 0, AGG_MIS_CAP, AGG_LOOP_CAP, AGG_RESTRICT_CAP, AGG_STALLED };

// The order of the next level (what old_mis forms from the partitions), for the weighted
// graph's kernel to write: the graph's nodes are aggregates, with their member nodes.
struct OrderArgs {
  const int32_t *astart, *members;  // members of aggregate a: members[astart[a] .. astart[a + 1])
  int32_t *part_idx, *old_of, *new_id, *agg_idx, *xadj_out, *adj_out, *iperm, *perm, *agg_of, *part_of_row;
};

struct AggArgs {
  int n;
  const int32_t *xadj, *adj, *w;  // w: node weights (weighted graph), else null
  const uint32_t* seeds;
  int depth, min_size, max_size, full_size;
  uint32_t* rnd;                // n
  unsigned long long *k0, *k1;  // n each; k0 also holds the partitions' best moves
  int32_t *mis, *part, *pout, *sizes, *map, *to;  // n each
  int32_t* res;  // status, parts after the removals, largest label + 1, 1 when the labels are in pout
  OrderArgs o;   // weighted graph: part_idx and the rest, else null pointers
};

// Exchanges one value per CTA; v[r] = CTA r's value on return.  Two buffers: a value is
// overwritten two exchanges later, when every CTA has passed the barrier between.
struct ClusterExchange {
  int (*buf)[kAggCtas];
  int turn = 0, C, me;
  __device__ const int* operator()(cg::cluster_group& cl, int value) {
    __syncthreads();
    if ((int)threadIdx.x < C) *cl.map_shared_rank(&buf[turn][me], threadIdx.x) = value;
    cl.sync();
    const int* v = buf[turn];
    turn ^= 1;
    return v;
  }
  __device__ int sum(cg::cluster_group& cl, int value) {
    const int* v = (*this)(cl, value);
    int t = 0;
    for (int r = 0; r < C; r++) t += v[r];
    return t;
  }
  __device__ int max(cg::cluster_group& cl, int value) {
    const int* v = (*this)(cl, value);
    int t = v[0];
    for (int r = 1; r < C; r++) t = ::max(t, v[r]);
    return t;
  }
  // (sum of the lower CTAs' values, sum of all)
  __device__ int2 prefix(cg::cluster_group& cl, int value) {
    const int* v = (*this)(cl, value);
    int lower = 0, all = 0;
    for (int r = 0; r < C; r++) {
      if (r < me) lower += v[r];
      all += v[r];
    }
    return make_int2(lower, all);
  }
};

// Sum (or maximum) of one value per thread; the result in every thread.
__device__ __forceinline__ int agg_block_sum(int v, int* sh) {
  v = __reduce_add_sync(0xffffffffu, v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  return __reduce_add_sync(0xffffffffu, sh[threadIdx.x & 31]);
}
__device__ __forceinline__ int agg_block_max(int v, int* sh) {
  v = __reduce_max_sync(0xffffffffu, v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  const int l = threadIdx.x & 31;
  return __reduce_max_sync(0xffffffffu, l < (int)(blockDim.x >> 5) ? sh[l] : INT32_MIN);
}
// Inclusive prefix of a flag over the block, in thread order; *total gets the block's count.
__device__ __forceinline__ int agg_block_rank(bool flag, int* sh, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned m = __ballot_sync(0xffffffffu, flag);
  __syncthreads();
  if (lane == 0) sh[warp] = __popc(m);
  __syncthreads();
  const int mine = sh[lane];
  *total = (int)__reduce_add_sync(0xffffffffu, mine);
  const int below = (int)__reduce_add_sync(0xffffffffu, lane < warp ? mine : 0);
  return below + __popc(m & (0xffffffffu >> (31 - lane)));
}

// Exclusive prefix of one value per thread over the block; *total gets the block's sum.
__device__ __forceinline__ int agg_block_scan(int v, int* sh, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  __syncthreads();
  if (lane == 31) sh[warp] = x;
  __syncthreads();
  const int mine = sh[lane];
  *total = (int)__reduce_add_sync(0xffffffffu, mine);
  const int below = (int)__reduce_add_sync(0xffffffffu, lane < warp ? mine : 0);
  return below + x - v;
}

// Arrays that other CTAs write are read from L2 (__ldcg): a line of this SM's L1 may be old.
__global__ void __launch_bounds__(kAggThreads) aggregate_cluster_kernel(AggArgs a) {
  __shared__ int xbuf[2][kAggCtas];
  __shared__ int sh[32];
  cg::cluster_group cl = cg::this_cluster();
  ClusterExchange x{xbuf};
  x.C = (int)cl.num_blocks();
  x.me = (int)cl.block_rank();
  const int n = a.n, tid = threadIdx.x;
  const int per = (n + x.C - 1) / x.C, lo = min(n, x.me * per), hi = min(n, lo + per);
  const int32_t* __restrict__ xadj = a.xadj;
  const int32_t* __restrict__ adj = a.adj;
  int status = AGG_OK;
  // ---- randomized MIS: rounds of `depth` propagations until every node is decided
  unsigned long long *ki = a.k0, *ko = a.k1;
  for (int round = 0;; round++) {
    if (round >= kCap) {
      status = AGG_MIS_CAP;
      break;
    }
    for (int i = lo + tid; i < hi; i += kAggThreads) {
      uint32_t z;
      if (round == 0) {
        z = a.seeds[i & 32767];
        for (int t = 0; t <= i >> 15; t++) z = taus(z);
        ki[i] = mis_key((int32_t)(z % 1000000u), i);
      } else {
        z = taus(a.rnd[i]);
        const int st = a.mis[i];
        ki[i] = mis_key(st == -1 ? (int32_t)(z % 1000000u) : (st == 1 ? 1000001 : 0), i);
      }
      a.rnd[i] = z;
    }
    cl.sync();
    int undecided = 0;
    for (int it = 0; it < a.depth; it++) {
      for (int i = lo + tid; i < hi; i += kAggThreads) {
        unsigned long long k = ki[i];
        if ((k >> 32) < 1000001u) {
          const int e1 = xadj[i + 1];
          for (int e0 = xadj[i]; e0 < e1; e0 += 8) {
            int nb[8];
            unsigned long long kn[8];
#pragma unroll
            for (int q = 0; q < 8; q++) nb[q] = e0 + q < e1 ? adj[e0 + q] : i;
#pragma unroll
            for (int q = 0; q < 8; q++) kn[q] = __ldcg(ki + nb[q]);
#pragma unroll
            for (int q = 0; q < 8; q++)
              if ((kn[q] >> 32) > 0u && kn[q] > k) k = kn[q];
          }
        }
        ko[i] = k;
        if (it == a.depth - 1) {
          const int best = (int)(k >> 32), org = (int)(uint32_t)k;
          const int st = org == i ? 1 : best == 1000001 ? 0 : -1;
          a.mis[i] = st;
          undecided |= st == -1;
        }
      }
      unsigned long long* t = ki;
      ki = ko;
      ko = t;
      if (it < a.depth - 1) cl.sync();
    }
    if (x.sum(cl, __syncthreads_or(undecided)) == 0) break;
  }
  // ---- labels: the MIS nodes numbered in order
  int32_t *pin = a.part, *po = a.pout;
  int count;
  {
    int ones = 0;
    for (int i = lo + tid; i < hi; i += kAggThreads) ones += a.mis[i] == 1;
    const int2 pre = x.prefix(cl, agg_block_sum(ones, sh));
    count = pre.y;
    int base = pre.x;
    for (int i0 = lo; i0 < hi; i0 += kAggThreads) {
      const int i = i0 + tid;
      const bool root = i < hi && a.mis[i] == 1;
      int total;
      const int rank = agg_block_rank(root, sh, &total);
      if (i < hi) pin[i] = root ? base + rank - 1 : -1;
      base += total;
    }
  }
  cl.sync();
  bool first = true;
  for (int loop = 0; status == AGG_OK; loop++) {
    if (loop >= kCap) {
      status = AGG_LOOP_CAP;
      break;
    }
    // ---- allocation passes: each node without a part takes its first labelled neighbour's
    for (;;) {
      int left = 0, changed = 0;
      for (int i = lo + tid; i < hi; i += kAggThreads) {
        int p = pin[i];
        if (p == -1) {
          const int e1 = xadj[i + 1];
          for (int e0 = xadj[i]; e0 < e1 && p == -1; e0 += 8) {
            int nb[8], cnd[8];
#pragma unroll
            for (int q = 0; q < 8; q++) nb[q] = e0 + q < e1 ? adj[e0 + q] : -1;
#pragma unroll
            for (int q = 0; q < 8; q++) cnd[q] = nb[q] >= 0 ? __ldcg(pin + nb[q]) : -1;
#pragma unroll
            for (int q = 0; q < 8; q++)
              if (p == -1 && cnd[q] != -1) p = cnd[q];
          }
          if (p != -1) changed = 1;
          else left = 1;
        }
        po[i] = p;
      }
      int32_t* t = pin;
      pin = po;
      po = t;
      // nodes are left and none joined: bit 0 of any CTA set, bit 1 of none
      const int* v = x(cl, (__syncthreads_or(left) ? 1 : 0) | (__syncthreads_or(changed) ? 2 : 0));
      int any = 0;
      for (int r = 0; r < x.C; r++) any |= v[r];
      if (!(any & 1)) break;
      if (!(any & 2)) {
        status = AGG_STALLED;
        break;
      }
    }
    if (status != AGG_OK) break;
    const bool restrict_now = a.w && (!first || count < 10);
    // ---- sizes (weights) of the parts
    const int pper = (count + x.C - 1) / x.C, plo = min(count, x.me * pper), phi = min(count, plo + pper);
    for (int p = plo + tid; p < phi; p += kAggThreads) {
      a.sizes[p] = 0;
      if (restrict_now) a.k0[p] = 0ull;
    }
    cl.sync();
    for (int i = lo + tid; i < hi; i += kAggThreads) atomicAdd(&a.sizes[pin[i]], a.w ? a.w[i] : 1);
    cl.sync();
    if (restrict_now) {
      // ---- partitions above max_size give nodes away, one per round
      const int opt = a.full_size / count;
      for (int loops = 0;; loops++) {
        int m = INT32_MIN;
        for (int p = plo + tid; p < phi; p += kAggThreads) m = max(m, __ldcg(a.sizes + p));
        if (x.max(cl, agg_block_max(m, sh)) <= a.max_size) break;
        if (loops >= kCap) {
          status = AGG_RESTRICT_CAP;
          break;
        }
        for (int i = lo + tid; i < hi; i += kAggThreads) {
          int cur, add;
          const unsigned long long key = desirability<true>(i, opt, xadj, adj, pin, a.sizes, a.w, cur, add);
          a.to[i] = add;
          atomicMax(&a.k0[cur], key);
        }
        cl.sync();
        for (int p = plo + tid; p < phi; p += kAggThreads) {
          const unsigned long long key = __ldcg(a.k0 + p);
          a.k0[p] = 0ull;
          const float d = __uint_as_float((unsigned)(key >> 32));
          const int idx = (int)(key & 0xffffffffu);
          if ((double)d > .1) {
            const int t = __ldcg(a.to + idx);
            __stcg(pin + idx, t);
            atomicAdd(&a.sizes[t], a.w[idx]);
            atomicAdd(&a.sizes[p], -a.w[idx]);
          }
        }
        cl.sync();
      }
      break;
    }
    // ---- parts below the threshold dissolve, the others are renumbered in order
    int threshold = a.min_size;
    if (a.w) {
      first = false;
      const double avg = (double)a.full_size / count;
      threshold = (int)(avg * .7);
    }
    int small = 0;
    for (int p = plo + tid; p < phi; p += kAggThreads) small += __ldcg(a.sizes + p) < threshold;
    const int2 pre = x.prefix(cl, agg_block_sum(small, sh));
    if (pre.y == 0 && !a.w) break;
    int base = pre.x;
    for (int p0 = plo; p0 < phi; p0 += kAggThreads) {
      const int p = p0 + tid;
      const bool rm = p < phi && __ldcg(a.sizes + p) < threshold;
      int total;
      const int rank = agg_block_rank(rm, sh, &total);
      if (p < phi) a.map[p] = rm ? -1 : p - (base + rank);
      base += total;
    }
    count -= pre.y;
    cl.sync();
    for (int i = lo + tid; i < hi; i += kAggThreads) pin[i] = __ldcg(a.map + pin[i]);
    cl.sync();
  }
  int m = -1;
  for (int i = lo + tid; i < hi; i += kAggThreads) m = max(m, __ldcg(pin + i));
  m = x.max(cl, agg_block_max(m, sh));
  if (a.o.part_idx && status == AGG_OK) {
    // ---- aggregates ordered by (partition, id), their graph and their nodes renumbered
    const OrderArgs& o = a.o;
    const int npart = m + 1;
    const int pper = (npart + x.C - 1) / x.C, plo = min(npart, x.me * pper), phi = min(npart, plo + pper);
    const int warp = x.me * (kAggThreads / 32) + (tid >> 5), nwarps = x.C * (kAggThreads / 32), lane = tid & 31;
    for (int p = plo + tid; p < phi; p += kAggThreads) a.sizes[p] = a.map[p] = 0;
    cl.sync();
    for (int i = lo + tid; i < hi; i += kAggThreads) atomicAdd(&a.sizes[__ldcg(pin + i)], 1);
    cl.sync();
    {
      int mine = 0;
      for (int p = plo + tid; p < phi; p += kAggThreads) mine += __ldcg(a.sizes + p);
      int base = x.prefix(cl, agg_block_sum(mine, sh)).x;
      for (int p0 = plo; p0 < phi; p0 += kAggThreads) {
        const int p = p0 + tid;
        int total;
        const int before = agg_block_scan(p < phi ? __ldcg(a.sizes + p) : 0, sh, &total);
        if (p < phi) o.part_idx[p] = base + before;
        base += total;
      }
      if (x.me == 0 && tid == 0) o.part_idx[npart] = n;
    }
    cl.sync();
    for (int i = lo + tid; i < hi; i += kAggThreads) {
      const int p = __ldcg(pin + i);
      a.to[__ldcg(o.part_idx + p) + atomicAdd(&a.map[p], 1)] = i;
    }
    cl.sync();
    // a partition's aggregates in ascending order: each is placed by counting the smaller ones
    for (int p = warp; p < npart; p += nwarps) {
      const int b = __ldcg(o.part_idx + p), e = __ldcg(o.part_idx + p + 1);
      for (int q = b + lane; q < e; q += 32) {
        const int v = __ldcg(a.to + q);
        int rank = 0;
#pragma unroll 8
        for (int t = b; t < e; t++) rank += __ldcg(a.to + t) < v;
        o.old_of[b + rank] = v;
        o.new_id[v] = b + rank;
      }
    }
    cl.sync();
    {
      int nodes = 0, edges = 0;
      for (int q = lo + tid; q < hi; q += kAggThreads) {
        const int v = __ldcg(o.old_of + q);
        nodes += o.astart[v + 1] - o.astart[v];
        edges += xadj[v + 1] - xadj[v];
      }
      const int2 pn = x.prefix(cl, agg_block_sum(nodes, sh)), pe = x.prefix(cl, agg_block_sum(edges, sh));
      int bn = pn.x, be = pe.x;
      for (int q0 = lo; q0 < hi; q0 += kAggThreads) {
        const int q = q0 + tid;
        const int v = q < hi ? __ldcg(o.old_of + q) : 0;
        int tn, te;
        const int sn = agg_block_scan(q < hi ? o.astart[v + 1] - o.astart[v] : 0, sh, &tn);
        const int se = agg_block_scan(q < hi ? xadj[v + 1] - xadj[v] : 0, sh, &te);
        if (q < hi) {
          o.agg_idx[q] = bn + sn;
          o.xadj_out[q] = be + se;
        }
        bn += tn;
        be += te;
      }
      if (x.me == 0 && tid == 0) {
        o.agg_idx[n] = pn.y;
        o.xadj_out[n] = pe.y;
      }
    }
    cl.sync();
    for (int q = warp; q < n; q += nwarps) {
      const int v = __ldcg(o.old_of + q), p = __ldcg(pin + v);
      const int e0 = xadj[v], e1 = xadj[v + 1], eo = __ldcg(o.xadj_out + q);
      for (int e = e0 + lane; e < e1; e += 32) o.adj_out[eo + (e - e0)] = __ldcg(o.new_id + adj[e]);
      const int t0 = o.astart[v], t1 = o.astart[v + 1], no = __ldcg(o.agg_idx + q);
      for (int t = t0 + lane; t < t1; t += 32) {
        const int node = o.members[t], at = no + (t - t0);
        o.iperm[at] = node;
        o.perm[node] = at;
        o.agg_of[at] = q;
        o.part_of_row[at] = p;
      }
    }
  }
  if (x.me == 0 && tid == 0) {
    a.res[0] = status;
    a.res[1] = count;
    a.res[2] = m + 1;
    a.res[3] = pin == a.pout;
  }
  cl.sync();  // no CTA leaves while another may still write to its exchange buffers
}

// Runs aggregate_cluster_kernel: the labels in `part`, (parts after the removals, largest
// label + 1) in count and labels.
void aggregate_small(Ctx& c, int n, const int32_t* xadj, const int32_t* adj, int depth, int min_size, int max_size,
                     int full_size, const int32_t* weights, DBuf<int32_t>& part, int* count, int* labels,
                     const OrderArgs* order) {
  cudaStream_t s = c.stream;
  PhaseTimer pt(s, -4);
  DBuf<unsigned long long> keys((size_t)2 * n, s);
  DBuf<uint32_t> rnd(n, s);
  DBuf<int32_t> work((size_t)4 * n + 4, s), pout(n, s);
  part.alloc(n, s);
  AggArgs a{};
  a.n = n;
  a.xadj = xadj;
  a.adj = adj;
  a.w = weights;
  a.seeds = mis_seeds(c);
  a.depth = depth;
  a.min_size = min_size;
  a.max_size = max_size;
  a.full_size = full_size;
  a.rnd = rnd.p;
  a.k0 = keys.p;
  a.k1 = keys.p + n;
  a.part = part.p;
  a.pout = pout.p;
  a.res = work.p;
  a.mis = work.p + 4;
  a.sizes = a.mis + n;
  a.map = a.sizes + n;
  a.to = a.map + n;
  if (order) a.o = *order;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kAggThreads);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const int most = std::min(c.cluster_limit, largest_cluster(reinterpret_cast<const void*>(aggregate_cluster_kernel),
                                                             kAggThreads, kAggCtas));
  const int ctas = std::min(most, next_pow2((n + kAggThreads - 1) / kAggThreads));
  at[0].val.clusterDim.x = (unsigned)ctas;
  cfg.gridDim = dim3((unsigned)ctas);
  g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
  FG_CUDA(cudaLaunchKernelEx(&cfg, aggregate_cluster_kernel, a));
  int32_t h[4];
  FG_CUDA(cudaMemcpyAsync(h, a.res, sizeof(h), cudaMemcpyDeviceToHost, s));
  FG_CUDA(cudaStreamSynchronize(s));
  g_host_syncs.fetch_add(1, std::memory_order_relaxed);
  pt.mark("cluster");
  if (h[0] == AGG_MIS_CAP) throw Error(FEMGPU_ERR_LIMIT, "randomized MIS did not complete");
  if (h[0] == AGG_LOOP_CAP) throw Error(FEMGPU_ERR_LIMIT, "aggregation did not complete");
  if (h[0] == AGG_RESTRICT_CAP) throw Error(FEMGPU_ERR_LIMIT, "partition size restriction did not converge");
  if (h[0] == AGG_STALLED) throw_stalled();
  if (h[3]) std::swap(part, pout);
  *count = h[1];
  *labels = h[2];
}

// aggregateGraph / aggregateWeightedGraph (misHelpers.cu:513-677).  Returns the number
// of parts (the largest label + 1: the partition restriction of the weighted graph may
// empty a part).
// order (weighted graph only, or null): written too when the graph is aggregated by one
// kernel; *ordered tells.
int aggregate(Ctx& c, int n, int64_t edges, const int32_t* xadj, const int32_t* adj, int depth, bool weighted,
              int min_size, int max_size, int full_size, const int32_t* weights, DBuf<int32_t>& part,
              const OrderArgs* order = nullptr, bool* ordered = nullptr) {
  cudaStream_t s = c.stream;
  if (edges <= kClusterAggEdges && n <= kClusterAggEdges / 4 && depth > 0) {
    int count = 0, labels = 0;
    aggregate_small(c, n, xadj, adj, depth, min_size, max_size, full_size, weighted ? weights : nullptr, part, &count,
                    &labels, order);
    if (ordered) *ordered = order != nullptr;
    return weighted ? labels : count;
  }
  PhaseTimer pt(s, -4);
  DBuf<int32_t> mis;
  random_mis(c, n, xadj, adj, depth, mis);
  pt.mark("mis");
  DBuf<int32_t> incl(n + 1, s), aggregated(n, s), pout(n, s), counters(2, s);
  inclusive_scan(mis.p, incl.p, n, s);
  // the MIS size (= the number of parts, labelled 0 .. count-1 by label_roots_kernel)
  // comes back with the first allocation counters
  int mis_count = -1;
  part.alloc(n, s);
  FG_LAUNCH(label_roots_kernel, grid_for(n, 256), 256, 0, s, n, mis.p, incl.p, part.p, aggregated.p);
  bool first = true;
  for (int loop = 0;; loop++) {
    FG_REQUIRE(loop < kCap, FEMGPU_ERR_LIMIT, "aggregation did not complete");
    // two passes per host read: a pass after the one that leaves no node unallocated
    // changes nothing, and the counters describe the second pass
    for (int pass = 0; pass < 2; pass++) {
      counters.zero();
      FG_LAUNCH(allocate_kernel, grid_for(n, 256), 256, 0, s, n, xadj, adj, part.p, pout.p, aggregated.p,
                counters.p);
      std::swap(part, pout);
    }
    int32_t h[2];
    counters.download(h, 2);
    if (mis_count < 0 && n > 0) FG_CUDA(cudaMemcpyAsync(&mis_count, incl.p + (n - 1), sizeof(int32_t),
                                                       cudaMemcpyDeviceToHost, s));
    FG_CUDA(cudaStreamSynchronize(s));
    g_host_syncs.fetch_add(1, std::memory_order_relaxed);
    if (mis_count < 0) mis_count = 0;
    pt.mark("allocate");
    if (h[0] == 0) {
      if (!weighted) {
        // unweighted parts are never emptied: their count is tracked, not read back
        const int removed = remove_small_parts(c, n, part, nullptr, 0, min_size, full_size, aggregated, mis_count);
        if (removed == 0) return mis_count;
        mis_count -= removed;
      } else {
        // the labels are still contiguous and non-empty here (the restriction below may
        // empty a partition, but nothing reads the count after it): tracked, not read
        if (!first || mis_count < 10) {
          restrict_partitions(c, max_size, full_size, n, xadj, adj, part, weights, mis_count);
          return reduce_max(part.p, n, s) + 1;
        }
        first = false;
        mis_count -= remove_small_parts(c, n, part, weights, 1, 0, full_size, aggregated, mis_count);
      }
    } else if (h[1] == 0) {
      // also the case where every aggregate was removed as undersized (the reference
      // loops forever there)
      throw_stalled();
    }
  }
}

__global__ void scatter_bucket_kernel(int n, const int32_t* key, const int32_t* start, int32_t* cursor, int32_t* out) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    int k = key[i];
    out[start[k] + atomicAdd(&cursor[k], 1)] = i;
  }
}

__global__ void node_degree_to_agg_kernel(int n, const int32_t* xadj, const int32_t* fine, int32_t* cnt) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) atomicAdd(&cnt[fine[i]], xadj[i + 1] - xadj[i]);
}

// Degree of each member node, in member order (aggregates in order, members ascending).
__global__ void member_degree_kernel(int n, const int32_t* members, const int32_t* xadj, int32_t* deg) {
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < n) deg[q] = xadj[members[q] + 1] - xadj[members[q]];
}

// Induced-graph rows by hashing: one warp per aggregate walks the flattened neighbour
// lists of its members 32 entries at a time (flat index f of member q starts at
// noff[q]), groups equal aggregate ids with __match_any_sync, inserts each new id once
// into a shared-memory set and finally sorts the set, so a row holds the sorted distinct
// neighbour aggregates (what sorting the candidate list and dropping duplicates gives).
// An aggregate with more than kIndCap - 32 distinct neighbours sets *overflow.
constexpr int kIndCap = 256;

__device__ __forceinline__ unsigned induced_hash(unsigned b) { return (b * 2654435761u) >> 9; }

__global__ void __launch_bounds__(256) induced_hash_kernel(int nagg, const int32_t* __restrict__ astart,
                                                           const int32_t* __restrict__ members,
                                                           const int32_t* __restrict__ noff,
                                                           const int32_t* __restrict__ xadj,
                                                           const int32_t* __restrict__ adj,
                                                           const int32_t* __restrict__ fine, int32_t* tmp,
                                                           int32_t* ucount, int32_t* overflow) {
  __shared__ int32_t hk[8][kIndCap];
  __shared__ int32_t sk[8][kIndCap];
  __shared__ int s_cnt[8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int a = blockIdx.x * 8 + w; a < nagg; a += gridDim.x * 8) {
    for (int t = lane; t < kIndCap; t += 32) hk[w][t] = -1;
    if (lane == 0) s_cnt[w] = 0;
    __syncwarp();
    const int q0 = astart[a], q1 = astart[a + 1];
    const int f0 = noff[q0], f1 = noff[q1];
    bool over = false;
    for (int fb = f0; fb < f1 && !over; fb += 32) {
      const int f = fb + lane;
      int b = -1;
      if (f < f1) {
        int lo = q0, hi = q1 - 1;  // last member q with noff[q] <= f
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (noff[mid] <= f) lo = mid;
          else hi = mid - 1;
        }
        const int i = members[lo];
        b = fine[adj[xadj[i] + (f - noff[lo])]];
        if (b == a) b = -1;
      }
      const unsigned peers = __match_any_sync(0xffffffffu, b);
      if (b >= 0 && (__ffs(peers) - 1) == lane) {
        unsigned slot = induced_hash((unsigned)b) & (kIndCap - 1);
        for (int p = 0; p < kIndCap; p++) {
          const int prev = atomicCAS(&hk[w][slot], -1, b);
          if (prev == -1) {
            atomicAdd(&s_cnt[w], 1);
            break;
          }
          if (prev == b) break;
          slot = (slot + 1) & (kIndCap - 1);
        }
      }
      __syncwarp();
      over = s_cnt[w] > kIndCap - 32;  // the next chunk might not fit
    }
    if (over) {
      if (lane == 0) *overflow = 1;
      continue;
    }
    // compact the set, pad to a power of two, sort
    const int cnt = s_cnt[w];
    int base = 0;
    for (int t0 = 0; t0 < kIndCap; t0 += 32) {
      const int key = hk[w][t0 + lane];
      const unsigned m = __ballot_sync(0xffffffffu, key >= 0);
      if (key >= 0) sk[w][base + __popc(m & ((1u << lane) - 1u))] = key;
      base += __popc(m);
    }
    const int np2 = next_pow2(cnt < 2 ? 2 : cnt);
    for (int t = cnt + lane; t < np2; t += 32) sk[w][t] = INT32_MAX;
    __syncwarp();
    bitonic_sort_shared(sk[w], np2, lane, 32, WarpSync());
    for (int t = lane; t < cnt; t += 32) tmp[(int64_t)a * kIndCap + t] = sk[w][t];
    if (lane == 0) ucount[a] = cnt;
    __syncwarp();
  }
}

// Rows of fixed stride `stride` in src to their offsets doff in dst, one warp per row.
__global__ void compact_stride_kernel(int nseg, const int32_t* src, int stride, const int32_t* doff, int32_t* dst) {
  const int lane = threadIdx.x & 31;
  for (int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < nseg; k += (gridDim.x * blockDim.x) >> 5) {
    const int len = doff[k + 1] - doff[k];
    for (int t = lane; t < len; t += 32) dst[doff[k] + t] = src[(int64_t)k * stride + t];
  }
}

// One thread per member node: the aggregates of its neighbours go to the node's slice
// of its aggregate's candidate list (its own aggregate as INT32_MAX padding), so every
// list holds the same multiset as a member-by-member walk.
__global__ void induced_candidates_nodes_kernel(int n, const int32_t* members, const int32_t* noff,
                                                const int32_t* __restrict__ xadj, const int32_t* __restrict__ adj,
                                                const int32_t* __restrict__ fine, int32_t* cand) {
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const int i = members[q], a = fine[i];
  int o = noff[q];
  for (int e = xadj[i]; e < xadj[i + 1]; e++) {
    const int b = fine[adj[e]];
    cand[o++] = b != a ? b : INT32_MAX;
  }
}

__global__ void drop_padding_kernel(int nseg, const int32_t* off, int32_t* cnt, const int32_t* vals) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < nseg && cnt[k] > 0 && vals[off[k] + cnt[k] - 1] == INT32_MAX) cnt[k]--;
}

__global__ void compact_segments_kernel(int nseg, const int32_t* src, const int32_t* soff, const int32_t* doff,
                                        int32_t* dst) {
  int lane = threadIdx.x & 31;
  for (int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < nseg; k += (gridDim.x * blockDim.x) >> 5) {
    int len = doff[k + 1] - doff[k];
    for (int t = lane; t < len; t += 32) dst[doff[k] + t] = src[soff[k] + t];
  }
}

__global__ void invert_kernel(int n, const int32_t* order, int32_t* inv) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) inv[order[i]] = i;
}

__global__ void gather_len_kernel(int n, const int32_t* order, const int32_t* off, int32_t* len) {
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < n) len[q] = off[order[q] + 1] - off[order[q]];
}

__global__ void remap_graph_kernel(int nagg, const int32_t* old_of, const int32_t* ixadj, const int32_t* iadj,
                                   const int32_t* new_id, const int32_t* xo, int32_t* ao) {
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nagg) return;
  int a = old_of[q];
  int o = xo[q];
  for (int e = ixadj[a]; e < ixadj[a + 1]; e++) ao[o++] = new_id[iadj[e]];
}

__global__ void node_order_kernel(int nagg, const int32_t* old_of, const int32_t* astart, const int32_t* members,
                                  const int32_t* agg_idx, const int32_t* coarse, int32_t* iperm, int32_t* agg_of,
                                  int32_t* part_of_row) {
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nagg) return;
  int a = old_of[q];
  int o = agg_idx[q];
  int p = coarse[a];
  for (int t = astart[a]; t < astart[a + 1]; t++) {
    iperm[o] = members[t];
    agg_of[o] = q;
    part_of_row[o] = p;
    o++;
  }
}

// Opt-in setup phase timing (environment FEMGPU_PROFILE set): synchronizes between
// phases and prints the host wall time of each to stderr.

struct OldMisOut {
  int nagg = 0, npart = 0;
  DBuf<int32_t> perm, iperm, agg_idx, part_idx, agg_of, part_of_row, xadj_out, adj_out;
  int64_t nnz_out = 0;
};

// misHelpers::CP::OldMIS (ComputePermutationMethods.cu:22-151).
void old_mis(Ctx& c, int n, int64_t edges, const int32_t* xadj, const int32_t* adj, OldMisOut& o) {
  cudaStream_t s = c.stream;
  const int params = c.cfg.randMisParameters;
  const int fine_depth = params % 100, coarse_depth = (params / 100) % 100, min_agg = (params / 10000) % 10;
  PhaseTimer pt(s, -1);
  DBuf<int32_t> fine;
  const int nagg = aggregate(c, n, edges, xadj, adj, fine_depth, false, min_agg, 0, n, nullptr, fine);
  pt.mark("fine agg");
  // aggregate member lists, ascending node id
  DBuf<int32_t> acount(nagg + 1, s), astart(nagg + 1, s), cursor(nagg, s), members(n, s);
  acount.zero();
  FG_LAUNCH(histogram_kernel, grid_for(n, 256), 256, 0, s, n, fine.p, nullptr, acount.p);
  exclusive_scan_async(acount.p, astart.p, nagg, s);
  cursor.zero();
  FG_LAUNCH(scatter_bucket_kernel, grid_for(n, 256), 256, 0, s, n, fine.p, astart.p, cursor.p, members.p);
  segmented_sort_i32(members.p, astart.p, nagg, nullptr, s);
  // induced graph (getInducedGraph, misHelpers.cu:1078-1107): sorted unique neighbour aggregates
  DBuf<int32_t> ucount(nagg + 1, s), ixadj(nagg + 1, s), iadj;
  DBuf<int32_t> mdeg(n + 1, s), noff(n + 1, s);
  FG_LAUNCH(member_degree_kernel, grid_for(n, 256), 256, 0, s, n, members.p, xadj, mdeg.p);
  exclusive_scan_async(mdeg.p, noff.p, n, s);
  bool induced_done = false;
  int64_t induced_nnz = 0;
  {
    DBuf<int32_t> tmp((size_t)nagg * kIndCap, s), ovf(1, s);
    ovf.zero();
    FG_LAUNCH(induced_hash_kernel, (int)std::min<int64_t>((nagg + 7) / 8, 152 * 16), 256, 0, s, nagg, astart.p,
              members.p, noff.p, xadj, adj, fine.p, tmp.p, ucount.p, ovf.p);
    // the overflow flag and the total come back in one round trip
    exclusive_scan_async(ucount.p, ixadj.p, nagg, s);
    int32_t h_ovf = 0, h_tot = 0;
    FG_CUDA(cudaMemcpyAsync(&h_ovf, ovf.p, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    FG_CUDA(cudaMemcpyAsync(&h_tot, ixadj.p + nagg, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    FG_CUDA(cudaStreamSynchronize(s));
    g_host_syncs.fetch_add(1, std::memory_order_relaxed);
    if (h_ovf == 0) {
      const int64_t innz = h_tot;
      induced_nnz = innz;
      iadj.alloc(innz > 0 ? innz : 1, s);
      FG_LAUNCH(compact_stride_kernel, grid_for((int64_t)nagg * 32, 256), 256, 0, s, nagg, tmp.p, kIndCap, ixadj.p,
                iadj.p);
      induced_done = true;
    }
  }
  if (!induced_done) {
    // an aggregate with more than kIndCap neighbour aggregates: sort every candidate list
    DBuf<int32_t> ccount(nagg + 1, s), coff(nagg + 1, s);
    ccount.zero();
    FG_LAUNCH(node_degree_to_agg_kernel, grid_for(n, 256), 256, 0, s, n, xadj, fine.p, ccount.p);
    int64_t ncand = exclusive_scan(ccount.p, coff.p, nagg, s);
    DBuf<int32_t> cand(ncand > 0 ? ncand : 1, s);
    FG_LAUNCH(induced_candidates_nodes_kernel, grid_for(n, 256), 256, 0, s, n, members.p, noff.p, xadj, adj, fine.p,
              cand.p);
    segmented_sort_i32(cand.p, coff.p, nagg, ucount.p, s);
    FG_LAUNCH(drop_padding_kernel, grid_for(nagg, 256), 256, 0, s, nagg, coff.p, ucount.p, cand.p);
    int64_t innz = exclusive_scan(ucount.p, ixadj.p, nagg, s);
    induced_nnz = innz;
    iadj.alloc(innz > 0 ? innz : 1, s);
    FG_LAUNCH(compact_segments_kernel, grid_for((int64_t)nagg * 32, 256), 256, 0, s, nagg, cand.p, coff.p, ixadj.p,
              iadj.p);
  }
  pt.mark("induced");
  // partitions of aggregates (aggregateWeightedGraph, weights = aggregate sizes), then the
  // order of the next level: aggregates by (partition, old id), their graph with its rows in
  // that order and its entries renamed in place (remapInducedGraph, misHelpers.cu:1258-1280),
  // nodes by aggregate, members ascending.  Small graphs do it in the kernel that
  // partitions them (11 launches fewer).
  DBuf<int32_t> coarse, old_of(nagg, s), new_id(nagg, s);
  o.part_idx.alloc(nagg + 1, s);
  o.xadj_out.alloc(nagg + 1, s);
  o.nnz_out = induced_nnz;  // the same rows, reordered
  o.adj_out.alloc(o.nnz_out > 0 ? o.nnz_out : 1, s);
  o.agg_idx.alloc(nagg + 1, s);
  o.iperm.alloc(n, s);
  o.perm.alloc(n, s);
  o.agg_of.alloc(n, s);
  o.part_of_row.alloc(n, s);
  OrderArgs order{astart.p, members.p, o.part_idx.p, old_of.p, new_id.p, o.agg_idx.p, o.xadj_out.p,
                  o.adj_out.p, o.iperm.p, o.perm.p, o.agg_of.p, o.part_of_row.p};
  bool ordered = false;
  const int npart = aggregate(c, nagg, induced_nnz, ixadj.p, iadj.p, coarse_depth, true, 0, c.cfg.partitionMaxSize, n,
                              acount.p, coarse, &order, &ordered);
  o.part_idx.n = (size_t)npart + 1;  // (allocated for a partition per aggregate)
  pt.mark("partitions");
  if (!ordered) {
    DBuf<int32_t> pcount(npart + 1, s), pcur(npart, s), rlen(nagg + 1, s), asz(nagg + 1, s);
    pcount.zero();
    FG_LAUNCH(histogram_kernel, grid_for(nagg, 256), 256, 0, s, nagg, coarse.p, nullptr, pcount.p);
    exclusive_scan_async(pcount.p, o.part_idx.p, npart, s);
    pcur.zero();
    FG_LAUNCH(scatter_bucket_kernel, grid_for(nagg, 256), 256, 0, s, nagg, coarse.p, o.part_idx.p, pcur.p, old_of.p);
    segmented_sort_i32(old_of.p, o.part_idx.p, npart, nullptr, s);
    FG_LAUNCH(invert_kernel, grid_for(nagg, 256), 256, 0, s, nagg, old_of.p, new_id.p);
    FG_LAUNCH(gather_len_kernel, grid_for(nagg, 256), 256, 0, s, nagg, old_of.p, ixadj.p, rlen.p);
    exclusive_scan_async(rlen.p, o.xadj_out.p, nagg, s);
    FG_LAUNCH(remap_graph_kernel, grid_for(nagg, 256), 256, 0, s, nagg, old_of.p, ixadj.p, iadj.p, new_id.p,
              o.xadj_out.p, o.adj_out.p);
    FG_LAUNCH(gather_len_kernel, grid_for(nagg, 256), 256, 0, s, nagg, old_of.p, astart.p, asz.p);
    exclusive_scan_async(asz.p, o.agg_idx.p, nagg, s);
    FG_LAUNCH(node_order_kernel, grid_for(nagg, 256), 256, 0, s, nagg, old_of.p, astart.p, members.p, o.agg_idx.p,
              coarse.p, o.iperm.p, o.agg_of.p, o.part_of_row.p);
    FG_LAUNCH(invert_kernel, grid_for(n, 256), 256, 0, s, n, o.iperm.p, o.perm.p);
  }
  pt.mark("order");
  o.nagg = nagg;
  o.npart = npart;
}

// ---------------------------------------------------------------------------------
// Row-wise expand-sort-compress in shared memory.
//
// Each output row is generated as a list of (column, value) items in a fixed
// generation order, sorted stably by column, and every run of equal columns is
// summed left to right from its first item.  Modes:
//   PERMUTE  row i <- input row iperm[i], columns renamed by perm (no duplicates);
//   PROLONG  row i of Ap: items (agg_of[j], ((-omega) a_ij) / d_i), then (agg_of[i], 1)
//            (generateProlongatorFull_d, smoothedMG_amg_level.cu:321-387);
//   SPGEMM   row i of A*B: items (k, a_ij b_jk) for j ascending, then k ascending
//            (the product of generateNextLevelMatrixFull_d, :390-400).
// Pass 0 writes per-row item counts, pass 1 unique counts, pass 2 the row.
enum EscMode { ESC_PERMUTE = 0, ESC_PROLONG = 1, ESC_SPGEMM = 2 };

template <class T>
struct EscArgs {
  int n;
  const int32_t* arp;
  const int32_t* aci;
  const T* av;
  const int32_t* brp;
  const int32_t* bci;
  const T* bv;
  const int32_t* perm;   // PERMUTE: old->new column map (nullptr = identity)
  const int32_t* iperm;  // PERMUTE: output row -> input row (nullptr = identity)
  const int32_t* agg_of; // PROLONG
  const T* diag;         // PROLONG
  T neg_omega;           // PROLONG
  const int32_t* big_rows;  // block tier: list of rows
  int nbig;
  int32_t* counts;       // pass 0/1 output
  const int32_t* orp;    // pass 2: output row offsets
  int32_t* oci;
  T* ov;
  int32_t* overflow;
  int thread_cap;        // rows with at most this many items use the thread tier
  int64_t known_nnz;     // PERMUTE: the input's entry count (every entry is kept), else 0
  int max_items;         // bound on a row's items when known, else 0
};

constexpr int kEscWarpCap = 1024;
constexpr int kEscWarps = 4;
constexpr int kEscBlockCap = 8192;
constexpr int kEscBlockThreads = 512;

template <class T, int MODE>
__device__ __forceinline__ int esc_input_row(const EscArgs<T>& a, int i) {
  return (MODE == ESC_PERMUTE && a.iperm) ? a.iperm[i] : i;
}

// Number of items of row i.
template <class T, int MODE>
__device__ __forceinline__ int esc_row_items(const EscArgs<T>& a, int i) {
  int r = esc_input_row<T, MODE>(a, i);
  int b = a.arp[r], e = a.arp[r + 1];
  if (MODE == ESC_PERMUTE) return e - b;
  if (MODE == ESC_PROLONG) return e - b + 1;
  int s = 0;
  for (int q = b; q < e; q++) {
    int j = a.aci[q];
    s += a.brp[j + 1] - a.brp[j];
  }
  return s;
}

// Generates row i's items into keys (column << 32 | generation index) and vals.
// tid/nthr: cooperating threads; sync: their barrier.
template <class T, int MODE, class Sync>
__device__ void esc_generate(const EscArgs<T>& a, int i, unsigned long long* keys, T* vals, int tid, int nthr,
                             int* s_scan, Sync sync) {
  int r = esc_input_row<T, MODE>(a, i);
  int b = a.arp[r], e = a.arp[r + 1];
  if (MODE != ESC_SPGEMM) {
    for (int q = b + tid; q < e; q += nthr) {
      int g = q - b;
      int j = a.aci[q];
      int col;
      T v;
      if (MODE == ESC_PERMUTE) {
        col = a.perm ? a.perm[j] : j;
        v = a.av[q];
      } else {
        col = a.agg_of[j];
        T t = (a.neg_omega * a.av[q]) * (T)1;
        v = t / a.diag[i];
      }
      keys[g] = ((unsigned long long)(unsigned)col << 32) | (unsigned)g;
      vals[g] = v;
    }
    if (MODE == ESC_PROLONG && tid == 0) {
      int g = e - b;
      keys[g] = ((unsigned long long)(unsigned)a.agg_of[i] << 32) | (unsigned)g;
      vals[g] = (T)1;
    }
    return;
  }
  // SPGEMM: chunks of nthr A entries; offsets by an exclusive scan of B row lengths
  int base = 0;
  for (int c0 = b; c0 < e; c0 += nthr) {
    int q = c0 + tid;
    int len = 0, j = 0;
    if (q < e) {
      j = a.aci[q];
      len = a.brp[j + 1] - a.brp[j];
    }
    // block/warp exclusive scan of len via shared memory (nthr <= 512)
    s_scan[tid] = len;
    sync();
    for (int off = 1; off < nthr; off <<= 1) {
      int add = tid >= off ? s_scan[tid - off] : 0;
      sync();
      s_scan[tid] += add;
      sync();
    }
    int excl = s_scan[tid] - len;
    int total = s_scan[nthr - 1];
    sync();
    if (q < e) {
      T av = a.av[q];
      int jb = a.brp[j];
      for (int t = 0; t < len; t++) {
        int g = base + excl + t;
        keys[g] = ((unsigned long long)(unsigned)a.bci[jb + t] << 32) | (unsigned)g;
        vals[g] = av * a.bv[jb + t];
      }
    }
    base += total;
  }
}

// After sorting: count (pass 1) or write (pass 2) the reduced row.  Heads are the
// first item of each column run; each head's thread sums its run left to right.
// Heads are ranked by warp ballots plus an exclusive scan over the warps.
template <class T, class Sync>
__device__ int esc_reduce(const unsigned long long* keys, const T* vals_by_gen, int len, int tid, int nthr,
                          int* s_warp /* >= nthr/32 + 1 ints */, int32_t* oci, T* ov, bool write, Sync sync) {
  const int lane = tid & 31, w = tid >> 5, nw = (nthr + 31) >> 5;
  int total = 0;
  for (int c0 = 0; c0 < len; c0 += nthr) {
    const int p = c0 + tid;
    const bool head = p < len && (p == 0 || (keys[p] >> 32) != (keys[p - 1] >> 32));
    const unsigned m = __ballot_sync(0xffffffffu, head);
    int rank = __popc(m & ((1u << lane) - 1u)), chunk = __popc(m);
    if (nw > 1) {
      if (lane == 0) s_warp[w] = chunk;
      sync();
      if (tid == 0) {
        int t = 0;
        for (int k = 0; k < nw; k++) {
          int v = s_warp[k];
          s_warp[k] = t;
          t += v;
        }
        s_warp[nw] = t;
      }
      sync();
      rank += s_warp[w];
      chunk = s_warp[nw];
    }
    if (head && write) {
      const unsigned col = (unsigned)(keys[p] >> 32);
      T sum = vals_by_gen[(unsigned)(keys[p] & 0xffffffffu)];
      for (int q = p + 1; q < len && (unsigned)(keys[q] >> 32) == col; q++)
        sum = sum + vals_by_gen[(unsigned)(keys[q] & 0xffffffffu)];
      oci[total + rank] = (int32_t)col;
      ov[total + rank] = sum;
    }
    total += chunk;
    sync();
  }
  return total;
}

template <class T, int MODE>
__global__ void esc_count_items_kernel(EscArgs<T> a) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < a.n) a.counts[i] = esc_row_items<T, MODE>(a, i);
}

__global__ void collect_big_rows_kernel(int n, const int32_t* items, int cap, int hard_cap, int32_t* list,
                                        int32_t* nlist) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && items[i] > cap && items[i] <= hard_cap) list[atomicAdd(nlist, 1)] = i;
}

// Rows of more than thread_cap and at most kEscWarpCap items, one warp each.  A warp looks at
// `look` rows' item counts at a time: 32 on large levels (one row at a time, 2.1 M rows with
// none to sort took 0.4 ms per pass), few on small ones, whose rows need all the warps.  Items
// of a permuted row have distinct columns: up to kRankCap of them are placed by counting the
// smaller ones (a broadcast read and a compare per item and lane, no barriers) instead of a
// bitonic network: 80,338 rows of 100 items 406 -> 191 us.
constexpr int kRankCap = 256;

template <class T, int MODE, bool WRITE>
__global__ void esc_warp_kernel(EscArgs<T> a, const int32_t* __restrict__ items, int look) {
  extern __shared__ unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned long long* keys = reinterpret_cast<unsigned long long*>(smem_raw) + (size_t)w * kEscWarpCap;
  T* vals = reinterpret_cast<T*>(reinterpret_cast<unsigned long long*>(smem_raw) + (size_t)kEscWarps * kEscWarpCap) +
            (size_t)w * kEscWarpCap;
  __shared__ int s_scan[kEscWarps][32];
  __shared__ int s_cnt[kEscWarps];
  for (int i0 = (blockIdx.x * kEscWarps + w) * look; i0 < a.n; i0 += gridDim.x * kEscWarps * look) {
    const int mylen = lane < look && i0 + lane < a.n ? items[i0 + lane] : 0;
    unsigned todo = __ballot_sync(0xffffffffu, mylen > a.thread_cap && mylen <= kEscWarpCap);
    while (todo) {
      const int src = __ffs(todo) - 1, i = i0 + src;
      todo &= todo - 1;
      const int len = __shfl_sync(0xffffffffu, mylen, src);
      if (MODE == ESC_PERMUTE && WRITE && len <= kRankCap) {
        const int r = esc_input_row<T, MODE>(a, i), rb = a.arp[r], out = a.orp[i];
        int32_t* col = reinterpret_cast<int32_t*>(keys);
        int32_t c[kRankCap / 32];
        int rank[kRankCap / 32];
#pragma unroll
        for (int q = 0; q < kRankCap / 32; q++) {
          const int g = lane + 32 * q;
          c[q] = INT32_MAX;
          rank[q] = 0;
          if (g < len) {
            const int j = a.aci[rb + g];
            c[q] = a.perm ? a.perm[j] : j;
          }
          col[g] = c[q];  // past the end INT32_MAX: never smaller
        }
        __syncwarp();
        auto count = [&](auto nq) {  // nq registers of 32 items cover the row
          for (int t = 0; t < len; t += 4) {
            const int4 o = *reinterpret_cast<const int4*>(col + t);
#pragma unroll
            for (int q = 0; q < decltype(nq)::value; q++)
              rank[q] += (o.x < c[q]) + (o.y < c[q]) + (o.z < c[q]) + (o.w < c[q]);
          }
        };
        if (len <= 64) count(std::integral_constant<int, 2>());
        else if (len <= 128) count(std::integral_constant<int, 4>());
        else count(std::integral_constant<int, 8>());
#pragma unroll
        for (int q = 0; q < kRankCap / 32; q++) {
          const int g = lane + 32 * q;
          if (g < len) {
            a.oci[out + rank[q]] = c[q];
            a.ov[out + rank[q]] = a.av[rb + g];
          }
        }
        __syncwarp();
        continue;
      }
      esc_generate<T, MODE>(a, i, keys, vals, lane, 32, s_scan[w], WarpSync());
      int np2 = next_pow2(len < 2 ? 2 : len);
      for (int p = len + lane; p < np2; p += 32) keys[p] = ~0ull;
      __syncwarp();
      bitonic_sort_shared(keys, np2, lane, 32, WarpSync());
      int out = WRITE ? a.orp[i] : 0;
      int cnt = esc_reduce<T>(keys, vals, len, lane, 32, &s_cnt[w], WRITE ? a.oci + out : nullptr,
                              WRITE ? a.ov + out : nullptr, WRITE, WarpSync());
      if (!WRITE && lane == 0) a.counts[i] = cnt;
      __syncwarp();
    }
  }
}

template <class T, int MODE, bool WRITE>
__global__ void esc_block_kernel(EscArgs<T> a, const int32_t* items) {
  extern __shared__ unsigned char smem_raw[];
  unsigned long long* keys = reinterpret_cast<unsigned long long*>(smem_raw);
  T* vals = reinterpret_cast<T*>(keys + kEscBlockCap);
  __shared__ int s_scan[kEscBlockThreads];
  __shared__ int s_cnt[kEscBlockThreads / 32 + 1];
  for (int b = blockIdx.x; b < a.nbig; b += gridDim.x) {
    int i = a.big_rows[b];
    int len = items[i];
    esc_generate<T, MODE>(a, i, keys, vals, threadIdx.x, blockDim.x, s_scan, BlockSync());
    int np2 = next_pow2(len);
    for (int p = len + threadIdx.x; p < np2; p += blockDim.x) keys[p] = ~0ull;
    __syncthreads();
    bitonic_sort_shared(keys, np2, threadIdx.x, blockDim.x, BlockSync());
    int out = WRITE ? a.orp[i] : 0;
    int cnt = esc_reduce<T>(keys, vals, len, threadIdx.x, blockDim.x, s_cnt, WRITE ? a.oci + out : nullptr,
                            WRITE ? a.ov + out : nullptr, WRITE, BlockSync());
    if (!WRITE && threadIdx.x == 0) a.counts[i] = cnt;
    __syncthreads();
  }
}

// Rows beyond the shared-memory sort capacity (they appear only on coarse levels,
// where the column count is small): one block per row, a dense accumulator over
// the output columns; thread 0 walks the items in generation order (so every
// column is summed left to right from its first item), then the block compacts
// the touched columns in ascending order.
template <class T, int MODE>
__device__ void esc_dense_row(const EscArgs<T>& a, int i, T* acc, unsigned char* mark, int ncols) {
  auto add = [&](int col, T v) {
    if (!mark[col]) {
      mark[col] = 1;
      acc[col] = v;
    } else {
      acc[col] = acc[col] + v;
    }
  };
  int r = esc_input_row<T, MODE>(a, i);
  int b = a.arp[r], e = a.arp[r + 1];
  for (int q = b; q < e; q++) {
    int j = a.aci[q];
    if (MODE == ESC_PERMUTE) {
      add(a.perm ? a.perm[j] : j, a.av[q]);
    } else if (MODE == ESC_PROLONG) {
      T t = (a.neg_omega * a.av[q]) * (T)1;
      add(a.agg_of[j], t / a.diag[i]);
    } else {
      T av = a.av[q];
      for (int f = a.brp[j]; f < a.brp[j + 1]; f++) add(a.bci[f], av * a.bv[f]);
    }
  }
  if (MODE == ESC_PROLONG) add(a.agg_of[i], (T)1);
}

template <class T, int MODE, bool WRITE>
__global__ void esc_dense_kernel(EscArgs<T> a, int ncols, T* gacc, unsigned char* gmark) {
  extern __shared__ unsigned char smem_raw[];
  const bool shared = gacc == nullptr;
  __shared__ int s_total;
  __shared__ int s_warp[32];
  for (int bi = blockIdx.x; bi < a.nbig; bi += gridDim.x) {
    int i = a.big_rows[bi];
    T* acc = shared ? reinterpret_cast<T*>(smem_raw) : gacc + (size_t)blockIdx.x * ncols;
    unsigned char* mark = shared ? smem_raw + (size_t)ncols * sizeof(T) : gmark + (size_t)blockIdx.x * ncols;
    for (int q = threadIdx.x; q < ncols; q += blockDim.x) mark[q] = 0;
    __syncthreads();
    if (threadIdx.x == 0) esc_dense_row<T, MODE>(a, i, acc, mark, ncols);
    __syncthreads();
    // ordered compaction of marked columns
    int base = 0;
    int out = WRITE ? a.orp[i] : 0;
    for (int c0 = 0; c0 < ncols; c0 += blockDim.x) {
      int q = c0 + threadIdx.x;
      int m = (q < ncols && mark[q]) ? 1 : 0;
      unsigned bal = __ballot_sync(0xffffffffu, m);
      int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
      if (lane == 0) s_warp[w] = __popc(bal);
      __syncthreads();
      if (threadIdx.x == 0) {
        int t = 0;
        for (int k = 0; k < (int)(blockDim.x >> 5); k++) {
          int v = s_warp[k];
          s_warp[k] = t;
          t += v;
        }
        s_total = t;
      }
      __syncthreads();
      if (m && WRITE) {
        int pos = base + s_warp[w] + __popc(bal & ((1u << lane) - 1u));
        a.oci[out + pos] = q;
        a.ov[out + pos] = acc[q];
      }
      base += s_total;
      __syncthreads();
    }
    if (!WRITE && threadIdx.x == 0) a.counts[i] = base;
    __syncthreads();
  }
}

__global__ void collect_dense_rows_kernel(int n, const int32_t* items, int cap, int32_t* list, int32_t* nlist) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && items[i] > cap) list[atomicAdd(nlist, 1)] = i;
}

// ---- thread tier: short PERMUTE / PROLONG rows, one thread per row -----------------
// Items are generated in order and merged into a sorted local list; a repeated
// column adds to its running sum (left to right from the first item).
constexpr int kThreadRowCap = 16;

// Bitonic network on N register-resident (key, value) pairs; every index is a
// compile-time constant after unrolling, so nothing spills to local memory.
template <class T, int N>
__device__ __forceinline__ void sort_network(unsigned long long (&k)[N], T (&v)[N]) {
#pragma unroll
  for (int size = 2; size <= N; size <<= 1) {
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
#pragma unroll
      for (int i = 0; i < N; i++) {
        const int j = i ^ stride;
        if (j > i) {
          const bool asc = (i & size) == 0;
          if ((k[i] > k[j]) == asc) {
            unsigned long long tk = k[i];
            k[i] = k[j];
            k[j] = tk;
            T tv = v[i];
            v[i] = v[j];
            v[j] = tv;
          }
        }
      }
    }
  }
}

template <class T, int MODE, bool WRITE>
__global__ void esc_thread_kernel(EscArgs<T> a, const int32_t* items) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  const int len = items[i];
  if (len > kThreadRowCap) return;
  unsigned long long key[kThreadRowCap];
  T val[kThreadRowCap];
  const int r = esc_input_row<T, MODE>(a, i);
  const int rb = a.arp[r], re = a.arp[r + 1];
#pragma unroll
  for (int g = 0; g < kThreadRowCap; g++) {
    key[g] = ~0ull;
    val[g] = (T)0;
    const int q = rb + g;
    if (q < re) {
      const int j = a.aci[q];
      int col;
      T v;
      if (MODE == ESC_PERMUTE) {
        col = a.perm ? a.perm[j] : j;
        v = a.av[q];
      } else {
        col = a.agg_of[j];
        T t = (a.neg_omega * a.av[q]) * (T)1;
        v = t / a.diag[i];
      }
      key[g] = ((unsigned long long)(unsigned)col << 32) | (unsigned)g;
      val[g] = v;
    } else if (MODE == ESC_PROLONG && q == re) {
      key[g] = ((unsigned long long)(unsigned)a.agg_of[i] << 32) | (unsigned)g;
      val[g] = (T)1;
    }
  }
  sort_network<T, kThreadRowCap>(key, val);
  // runs of equal columns summed left to right (generation order within the run)
  const int o = WRITE ? a.orp[i] : 0;
  int u = 0;
  unsigned cur = 0xffffffffu;
  T sum = (T)0;
#pragma unroll
  for (int g = 0; g < kThreadRowCap; g++) {
    if (key[g] == ~0ull) continue;
    const unsigned col = (unsigned)(key[g] >> 32);
    if (col != cur) {
      if (cur != 0xffffffffu) {
        if (WRITE) {
          a.oci[o + u] = (int32_t)cur;
          a.ov[o + u] = sum;
        }
        u++;
      }
      cur = col;
      sum = val[g];
    } else {
      sum = sum + val[g];
    }
  }
  if (cur != 0xffffffffu) {
    if (WRITE) {
      a.oci[o + u] = (int32_t)cur;
      a.ov[o + u] = sum;
    }
    u++;
  }
  if (!WRITE) a.counts[i] = u;
}

template <class T, int MODE>
void run_esc_sort(Ctx& c, EscArgs<T> a, int nrows_out, int ncols_out, DCsr<T>& out) {
  cudaStream_t s = c.stream;
  a.n = nrows_out;
  DBuf<int32_t> items(nrows_out + 1, s), ucnt, big, nbig, dense, ndense;
  if (MODE != ESC_PERMUTE) ucnt.alloc(nrows_out + 1, s);
  a.counts = items.p;
  FG_LAUNCH((esc_count_items_kernel<T, MODE>), grid_for(nrows_out, 256), 256, 0, s, a);
  // tiers above the thread's (warp, block, dense accumulator) run only where the longest
  // row's items, when the caller knows a bound, can reach them
  const bool warp_tier = a.max_items == 0 || a.max_items > kThreadRowCap;
  int32_t h_big = 0, h_dense = 0;
  if (a.max_items == 0 || a.max_items > kEscWarpCap) {
    big.alloc(nrows_out + 1, s);
    dense.alloc(nrows_out + 1, s);
    nbig.alloc(1, s);
    ndense.alloc(1, s);
    nbig.zero();
    ndense.zero();
    FG_LAUNCH(collect_big_rows_kernel, grid_for(nrows_out, 256), 256, 0, s, nrows_out, items.p, kEscWarpCap,
              kEscBlockCap, big.p, nbig.p);
    FG_LAUNCH(collect_dense_rows_kernel, grid_for(nrows_out, 256), 256, 0, s, nrows_out, items.p, kEscBlockCap,
              dense.p, ndense.p);
    // both counts in one round trip
    FG_CUDA(cudaMemcpyAsync(&h_big, nbig.p, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    FG_CUDA(cudaMemcpyAsync(&h_dense, ndense.p, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    FG_CUDA(cudaStreamSynchronize(s));
    g_host_syncs.fetch_add(1, std::memory_order_relaxed);
  }
  a.nbig = h_big;
  a.big_rows = big.p;
  EscArgs<T> ad = a;  // dense tier: rows with more items than the sort capacity
  ad.nbig = h_dense;
  ad.big_rows = dense.p;
  const int dgrid = std::min(ad.nbig, 152 * 2);
  const size_t dsm = (size_t)ncols_out * (sizeof(T) + 1);
  const bool dense_shared = dsm <= 200 * 1024;
  DBuf<T> gacc;
  DBuf<unsigned char> gmark;
  if (ad.nbig > 0 && !dense_shared) {
    FG_REQUIRE((size_t)dgrid * ncols_out * (sizeof(T) + 1) <= ((size_t)8 << 30), FEMGPU_ERR_LIMIT,
               "dense accumulator for long SpGEMM rows exceeds 8 GB");
    gacc.alloc((size_t)dgrid * ncols_out, s);
    gmark.alloc((size_t)dgrid * ncols_out, s);
  }
  if (ad.nbig > 0 && dense_shared) {
    ensure_smem(esc_dense_kernel<T, MODE, false>, dsm);
    ensure_smem(esc_dense_kernel<T, MODE, true>, dsm);
  }
  const size_t wsm = (size_t)kEscWarps * kEscWarpCap * (sizeof(unsigned long long) + sizeof(T));
  const size_t bsm = (size_t)kEscBlockCap * (sizeof(unsigned long long) + sizeof(T));
  if (warp_tier) {
    ensure_smem(esc_warp_kernel<T, MODE, false>, wsm);
    ensure_smem(esc_warp_kernel<T, MODE, true>, wsm);
  }
  if (a.nbig > 0) {
    ensure_smem(esc_block_kernel<T, MODE, false>, bsm);
    ensure_smem(esc_block_kernel<T, MODE, true>, bsm);
  }
  const int look = std::max(1, std::min(32, nrows_out / (152 * 64)));
  const int wgrid = (int)std::min<int64_t>(((int64_t)nrows_out + look * kEscWarps - 1) / (look * kEscWarps), 152 * 64);
  a.counts = ucnt.p;
  a.thread_cap = kThreadRowCap;
  // a permuted row has no repeated column: its output length is its item count, so the
  // counting pass is needed only for the prolongator
  if (MODE != ESC_PERMUTE) {
    FG_LAUNCH((esc_thread_kernel<T, MODE, false>), grid_for(nrows_out, 128), 128, 0, s, a, items.p);
    if (warp_tier) FG_LAUNCH((esc_warp_kernel<T, MODE, false>), wgrid, 32 * kEscWarps, wsm, s, a, items.p, look);
    if (a.nbig > 0)
      FG_LAUNCH((esc_block_kernel<T, MODE, false>), std::min(a.nbig, 152 * 2), kEscBlockThreads, bsm, s, a,
                items.p);
    if (ad.nbig > 0) {
      ad.counts = ucnt.p;
      FG_LAUNCH((esc_dense_kernel<T, MODE, false>), dgrid, 256, dense_shared ? dsm : 0, s, ad, ncols_out, gacc.p,
                gmark.p);
    }
  }
  out.n = nrows_out;
  out.m = ncols_out;
  out.rp.alloc(nrows_out + 1, s);
  if (MODE == ESC_PERMUTE && a.known_nnz > 0) {  // a permutation keeps every entry: no read-back
    exclusive_scan_async(items.p, out.rp.p, nrows_out, s);
    out.nnz = a.known_nnz;
  } else {
    out.nnz = exclusive_scan(MODE == ESC_PERMUTE ? items.p : ucnt.p, out.rp.p, nrows_out, s);
  }
  out.ci.alloc(out.nnz > 0 ? out.nnz : 1, s);
  out.v.alloc(out.nnz > 0 ? out.nnz : 1, s);
  a.orp = out.rp.p;
  a.oci = out.ci.p;
  a.ov = out.v.p;
  FG_LAUNCH((esc_thread_kernel<T, MODE, true>), grid_for(nrows_out, 128), 128, 0, s, a, items.p);
  if (warp_tier) FG_LAUNCH((esc_warp_kernel<T, MODE, true>), wgrid, 32 * kEscWarps, wsm, s, a, items.p, look);
  if (a.nbig > 0)
    FG_LAUNCH((esc_block_kernel<T, MODE, true>), std::min(a.nbig, 152 * 2), kEscBlockThreads, bsm, s, a, items.p);
  if (ad.nbig > 0) {
    ad.orp = out.rp.p;
    ad.oci = out.ci.p;
    ad.ov = out.v.p;
    FG_LAUNCH((esc_dense_kernel<T, MODE, true>), dgrid, 256, dense_shared ? dsm : 0, s, ad, ncols_out, gacc.p,
              gmark.p);
  }
}


// ---- hash SpGEMM: C = A B, row by row ----------------------------------------------
// A row's products are visited one A entry at a time; the entries of one B row have
// distinct columns, so every column receives at most one product per step and the
// threads of a step never touch the same accumulator.  Steps run in order, so each
// column is summed left to right in generation order starting from its first
// product -- the same value as the sort-based expand-sort-compress.  The unique
// columns are then sorted (bitonic, in shared memory) and written to the row's slot
// of a temporary buffer; rows whose unique count exceeds the table go to a larger
// tier.
constexpr int kHashWarpCap = 256;
constexpr int kHashWarps = 8;
constexpr int kHashBlockCap = 4096;
constexpr int kHashBlockThreads = 256;

__device__ __forceinline__ unsigned hash_col(unsigned c) { return (c * 2654435761u) >> 7; }

template <class T, class Sync>
__device__ bool hash_row_accumulate(const EscArgs<T>& a, int i, int32_t* hk, T* hv, int cap, int tid, int nth,
                                    int* s_flag, Sync sync) {
  for (int q = tid; q < cap; q += nth) hk[q] = -1;
  if (tid == 0) *s_flag = 0;
  sync();
  for (int e = a.arp[i]; e < a.arp[i + 1]; e++) {
    const int j = a.aci[e];
    const T av = a.av[e];
    const int fb = a.brp[j], fe = a.brp[j + 1];
    for (int f0 = fb; f0 < fe; f0 += nth) {
      const int f = f0 + tid;
      if (f < fe && *s_flag == 0) {
        const int col = a.bci[f];
        const T v = av * a.bv[f];
        unsigned slot = hash_col((unsigned)col) & (unsigned)(cap - 1);
        for (int probes = 0;; probes++) {
          if (probes >= cap) {
            *s_flag = 1;
            break;
          }
          int k = hk[slot];
          if (k == -1) {
            int prev = atomicCAS(&hk[slot], -1, col);
            if (prev == -1) {
              hv[slot] = v;
              break;
            }
            k = prev;
          }
          if (k == col) {
            hv[slot] = hv[slot] + v;
            break;
          }
          slot = (slot + 1) & (unsigned)(cap - 1);
        }
      }
      sync();
    }
  }
  return *s_flag == 0;
}

// Collects the occupied slots as (column << 32 | slot) keys, sorts them and writes
// the row; returns the unique count.  nth threads, warp-ballot compaction.
template <class T, class Sync>
__device__ int hash_row_emit(const int32_t* hk, const T* hv, unsigned long long* lst, int cap, int tid, int nth,
                             int* s_warp, int32_t* oci, T* ov, Sync sync) {
  const int lane = tid & 31, w = tid >> 5, nw = (nth + 31) >> 5;
  int total = 0;
  for (int c0 = 0; c0 < cap; c0 += nth) {
    const int q = c0 + tid;
    const bool occ = q < cap && hk[q] != -1;
    const unsigned m = __ballot_sync(0xffffffffu, occ);
    int rank = __popc(m & ((1u << lane) - 1u)), chunk = __popc(m);
    if (nw > 1) {
      if (lane == 0) s_warp[w] = chunk;
      sync();
      if (tid == 0) {
        int t = 0;
        for (int k = 0; k < nw; k++) {
          int v = s_warp[k];
          s_warp[k] = t;
          t += v;
        }
        s_warp[nw] = t;
      }
      sync();
      rank += s_warp[w];
      chunk = s_warp[nw];
    }
    if (occ) lst[total + rank] = ((unsigned long long)(unsigned)hk[q] << 32) | (unsigned)q;
    total += chunk;
    sync();
  }
  const int np2 = next_pow2(total < 2 ? 2 : total);
  for (int p = total + tid; p < np2; p += nth) lst[p] = ~0ull;
  sync();
  bitonic_sort_shared(lst, np2, tid, nth, sync);
  for (int p = tid; p < total; p += nth) {
    oci[p] = (int32_t)(lst[p] >> 32);
    ov[p] = hv[(unsigned)(lst[p] & 0xffffffffu)];
  }
  sync();
  return total;
}

// Warp tier: 32 products per step in generation order (A entries of the row taken 32
// at a time, their B rows flattened by a warp scan).  Lanes holding the same column
// are grouped with __match_any_sync; the group's lowest lane adds the group's
// products to the accumulator in lane order, so each column is still summed left
// to right in generation order.
template <class T>
__device__ bool hash_row_accumulate_matched(const EscArgs<T>& a, int i, int32_t* hk, T* hv, T* sv, int cap,
                                            int lane, int* s_flag) {
  for (int q = lane; q < cap; q += 32) hk[q] = -1;
  if (lane == 0) *s_flag = 0;
  __syncwarp();
  const int rb = a.arp[i], re = a.arp[i + 1];
  for (int eb = rb; eb < re; eb += 32) {
    const int e = eb + lane;
    int j = 0, len = 0;
    T av = (T)0;
    if (e < re) {
      j = a.aci[e];
      av = a.av[e];
      len = a.brp[j + 1] - a.brp[j];
    }
    int incl = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    const int jb = e < re ? a.brp[j] : 0;
    for (int g0 = 0; g0 < total; g0 += 32) {
      const int g = g0 + lane;
      const bool live = g < total;
      int owner = 0;
#pragma unroll
      for (int st = 16; st > 0; st >>= 1) {
        int probe = __shfl_sync(0xffffffffu, incl, owner + st - 1);
        if (probe <= g) owner += st;
      }
      owner = owner > 31 ? 31 : owner;
      const int o_incl = __shfl_sync(0xffffffffu, incl, owner);
      const int o_len = __shfl_sync(0xffffffffu, len, owner);
      const int o_jb = __shfl_sync(0xffffffffu, jb, owner);
      const T o_av = __shfl_sync(0xffffffffu, av, owner);
      int col = -1;
      T v = (T)0;
      if (live) {
        const int f = o_jb + (g - (o_incl - o_len));
        col = a.bci[f];
        v = o_av * a.bv[f];
      }
      sv[lane] = v;
      const unsigned peers = __match_any_sync(0xffffffffu, col);
      __syncwarp();
      const bool leader = live && (__ffs(peers) - 1) == lane;
      if (leader && *s_flag == 0) {
        unsigned slot = hash_col((unsigned)col) & (unsigned)(cap - 1);
        int found = -1;
        bool fresh = false;
        for (int probes = 0; probes < cap; probes++) {
          int k = hk[slot];
          if (k == -1) {
            int prev = atomicCAS(&hk[slot], -1, col);
            if (prev == -1) {
              found = (int)slot;
              fresh = true;
              break;
            }
            k = prev;
          }
          if (k == col) {
            found = (int)slot;
            break;
          }
          slot = (slot + 1) & (unsigned)(cap - 1);
        }
        if (found < 0) {
          *s_flag = 1;
        } else {
          unsigned m = peers;
          T acc = fresh ? sv[__ffs(m) - 1] : hv[found] + sv[__ffs(m) - 1];
          m &= m - 1;
          while (m) {
            acc = acc + sv[__ffs(m) - 1];
            m &= m - 1;
          }
          hv[found] = acc;
        }
      }
      __syncwarp();
    }
  }
  return *s_flag == 0;
}

// Galerkin-product rows with few distinct columns: one thread per row keeps up to
// kRowSlots (column, value) pairs in shared memory and adds every product to its
// column's slot in generation order (entries of the left row in order, each times
// the right row in order), the first product of a column starting its slot; rows
// with more distinct columns are listed for the warp tier.  Same sums as the hash
// tiers, sorted by column on output.
constexpr int kRowSlots = 32;
constexpr int kRowThreads = 128;

template <class T>
__global__ void __launch_bounds__(kRowThreads) spgemm_row_kernel(EscArgs<T> a, const int32_t* toff, int32_t* tci,
                                                                 T* tv, int32_t* counts, int32_t* over,
                                                                 int32_t* nover) {
  __shared__ int32_t sc[kRowSlots][kRowThreads];
  __shared__ T sv[kRowSlots][kRowThreads];
  const int t = threadIdx.x;
  const int i = blockIdx.x * blockDim.x + t;
  if (i >= a.n) return;
  int u = 0;
  bool overflow = false;
  const int ea = a.arp[i], eb = a.arp[i + 1];
  for (int e0 = ea; e0 < eb && !overflow; e0 += 8) {
    // 8 left entries at a time: their columns, values and right-row ranges are loaded
    // before the products (which then run in generation order)
    int kk[8], fb[8], fe[8];
    T avv[8];
#pragma unroll
    for (int q = 0; q < 8; q++) {
      kk[q] = e0 + q < eb ? a.aci[e0 + q] : 0;
      avv[q] = e0 + q < eb ? a.av[e0 + q] : (T)0;
    }
#pragma unroll
    for (int q = 0; q < 8; q++) {
      fb[q] = e0 + q < eb ? a.brp[kk[q]] : 0;
      fe[q] = e0 + q < eb ? a.brp[kk[q] + 1] : 0;
    }
    for (int m = 0; m < 8 && !overflow; m++)
    for (int f = fb[m]; f < fe[m]; f++) {
      const int j = a.bci[f];
      const T p = avv[m] * a.bv[f];
      int q = 0;
      while (q < u && sc[q][t] != j) q++;
      if (q < u) {
        sv[q][t] = sv[q][t] + p;
      } else if (u < kRowSlots) {
        sc[u][t] = j;
        sv[u][t] = p;
        u++;
      } else {
        overflow = true;
        break;
      }
    }
  }
  if (overflow) {
    over[atomicAdd(nover, 1)] = i;
    counts[i] = 0;
    return;
  }
  for (int q = 1; q < u; q++) {
    const int cj = sc[q][t];
    const T vj = sv[q][t];
    int p = q - 1;
    while (p >= 0 && sc[p][t] > cj) {
      sc[p + 1][t] = sc[p][t];
      sv[p + 1][t] = sv[p][t];
      p--;
    }
    sc[p + 1][t] = cj;
    sv[p + 1][t] = vj;
  }
  const int o = toff[i];
  for (int q = 0; q < u; q++) {
    tci[o + q] = sc[q][t];
    tv[o + q] = sv[q][t];
  }
  counts[i] = u;
}

// Rows `rows[0 .. *nrows)` (all rows when rows == nullptr), one warp per row.
template <class T>
__global__ void hash_warp_kernel(EscArgs<T> a, const int32_t* rows, const int32_t* nrows, const int32_t* toff,
                                 int32_t* tci, T* tv, int32_t* counts, int32_t* over, int32_t* nover) {
  __shared__ int32_t hk[kHashWarps][kHashWarpCap];
  __shared__ T hv[kHashWarps][kHashWarpCap];
  __shared__ unsigned long long lst[kHashWarps][kHashWarpCap];
  __shared__ T sv[kHashWarps][32];
  __shared__ int s_flag[kHashWarps];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int nr = rows ? *nrows : a.n;
  for (int ii = blockIdx.x * kHashWarps + w; ii < nr; ii += gridDim.x * kHashWarps) {
    const int i = rows ? rows[ii] : ii;
    bool ok = hash_row_accumulate_matched<T>(a, i, hk[w], hv[w], sv[w], kHashWarpCap, lane, &s_flag[w]);
    if (!ok) {
      if (lane == 0) {
        over[atomicAdd(nover, 1)] = i;
        counts[i] = 0;
      }
      __syncwarp();
      continue;
    }
    int u = hash_row_emit<T>(hk[w], hv[w], lst[w], kHashWarpCap, lane, 32, nullptr, tci + toff[i], tv + toff[i],
                             WarpSync());
    if (lane == 0) counts[i] = u;
    __syncwarp();
  }
}

template <class T>
__global__ void hash_block_kernel(EscArgs<T> a, const int32_t* rows, int nrows, const int32_t* toff, int32_t* tci,
                                  T* tv, int32_t* counts, int32_t* over, int32_t* nover) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned long long* lst = reinterpret_cast<unsigned long long*>(smem_raw);
  T* hv = reinterpret_cast<T*>(lst + kHashBlockCap);
  int32_t* hk = reinterpret_cast<int32_t*>(hv + kHashBlockCap);
  __shared__ int s_flag;
  __shared__ int s_warp[kHashBlockThreads / 32 + 1];
  for (int b = blockIdx.x; b < nrows; b += gridDim.x) {
    const int i = rows[b];
    bool ok = hash_row_accumulate<T>(a, i, hk, hv, kHashBlockCap, threadIdx.x, blockDim.x, &s_flag, BlockSync());
    if (!ok) {
      if (threadIdx.x == 0) {
        over[atomicAdd(nover, 1)] = i;
        counts[i] = 0;
      }
      __syncthreads();
      continue;
    }
    int u = hash_row_emit<T>(hk, hv, lst, kHashBlockCap, threadIdx.x, blockDim.x, s_warp, tci + toff[i],
                             tv + toff[i], BlockSync());
    if (threadIdx.x == 0) counts[i] = u;
    __syncthreads();
  }
}

// Galerkin-product rows of a narrow product (at most kDenseCols output columns, few
// rows): one warp per row with a dense accumulator over the output columns in shared
// memory.  The left row's entries are taken in order, and for each of them the lanes take
// the right row's entries, whose columns are distinct; so every column is summed in
// generation order, its first product starting the sum -- the sums of the hash tiers,
// without their probing.  Columns are listed as they are first hit, the list is sorted,
// and the row is written in ascending column order into its temporary slots.
constexpr int kDenseCols = 4096;
template <class T>
__host__ __device__ inline size_t dense_warp_smem(int ncols) {
  const size_t acc = ((size_t)ncols * sizeof(T) + 15) / 16 * 16;
  const size_t list = (size_t)next_pow2(ncols < 2 ? 2 : ncols) * sizeof(int32_t);
  const size_t mark = ((size_t)ncols + 15) / 16 * 16;
  return acc + list + mark;
}

template <class T>
__global__ void spgemm_dense_warp_kernel(EscArgs<T> a, int ncols, const int32_t* __restrict__ toff,
                                         int32_t* __restrict__ tci, T* __restrict__ tv, int32_t* __restrict__ counts) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const size_t per = dense_warp_smem<T>(ncols);
  unsigned char* base = smem_raw + (size_t)w * per;
  T* acc = reinterpret_cast<T*>(base);
  int32_t* list = reinterpret_cast<int32_t*>(base + ((size_t)ncols * sizeof(T) + 15) / 16 * 16);
  const int cap = next_pow2(ncols < 2 ? 2 : ncols);
  unsigned char* mark = reinterpret_cast<unsigned char*>(list + cap);
  for (int k = lane; k < ncols; k += 32) mark[k] = 0;
  __syncwarp();
  const unsigned below = (1u << lane) - 1u;
  // adds product v to column col (lanes hold distinct columns within one right row)
  int nt = 0;
  auto add = [&](bool live, int col, T v) {
    const bool fresh = live && mark[col] == 0;
    if (fresh) {
      mark[col] = 1;
      acc[col] = v;
    } else if (live) {
      acc[col] = acc[col] + v;
    }
    const unsigned m = __ballot_sync(0xffffffffu, fresh);
    if (fresh) list[nt + __popc(m & below)] = col;
    nt += __popc(m);
  };
  for (int i = blockIdx.x * nw + w; i < a.n; i += gridDim.x * nw) {
    nt = 0;
    const int qb = a.arp[i], qe = a.arp[i + 1];
    // the left row in chunks of 32 entries: lane t holds entry q0 + t's value and right
    // row bounds; each right row's first 32 entries are loaded one entry ahead
    for (int q0 = qb; q0 < qe; q0 += 32) {
      const int nq = min(32, qe - q0);
      T avq = (T)0;
      int bs = 0, be = 0;
      if (lane < nq) {
        const int j = a.aci[q0 + lane];
        avq = a.av[q0 + lane];
        bs = a.brp[j];
        be = a.brp[j + 1];
      }
      int b0 = __shfl_sync(0xffffffffu, bs, 0), b1 = __shfl_sync(0xffffffffu, be, 0);
      int ncol = b0 + lane < b1 ? a.bci[b0 + lane] : 0;
      T nval = b0 + lane < b1 ? a.bv[b0 + lane] : (T)0;
      for (int u = 0; u < nq; u++) {
        const T av = __shfl_sync(0xffffffffu, avq, u);
        const int c0 = ncol;
        const T v0 = nval;
        const int cb0 = b0, cb1 = b1;
        if (u + 1 < nq) {
          b0 = __shfl_sync(0xffffffffu, bs, u + 1);
          b1 = __shfl_sync(0xffffffffu, be, u + 1);
          ncol = b0 + lane < b1 ? a.bci[b0 + lane] : 0;
          nval = b0 + lane < b1 ? a.bv[b0 + lane] : (T)0;
        }
        add(cb0 + lane < cb1, c0, av * v0);
        __syncwarp();
        for (int f = cb0 + 32 + lane; f - lane < cb1; f += 32) {
          const bool live = f < cb1;
          add(live, live ? a.bci[f] : 0, live ? av * a.bv[f] : (T)0);
          __syncwarp();
        }
      }
    }
    const int np2 = next_pow2(nt < 2 ? 2 : nt);
    for (int t = nt + lane; t < np2; t += 32) list[t] = INT32_MAX;
    __syncwarp();
    bitonic_sort_shared(list, np2, lane, 32, WarpSync());
    const int o = toff ? toff[i] : i * ncols;  // without offsets a row's slots are a whole row
    for (int t = lane; t < nt; t += 32) {
      const int col = list[t];
      tci[o + t] = col;
      tv[o + t] = acc[col];
      mark[col] = 0;
    }
    if (lane == 0) counts[i] = nt;
    __syncwarp();
  }
}

__global__ void spgemm_capacity_kernel(int n, const int32_t* items, int ncols, int32_t* cap) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) cap[i] = min(items[i], ncols);
}

// Rows from their capacity-spaced temporary slots to the compact CSR: G lanes per row
// (G near the average row length, so short rows do not leave most of a warp idle).
template <class T, int G>
__global__ void compact_rows_copy_kernel(int n, const int32_t* toff, int stride, const int32_t* tci, const T* tv,
                                         const int32_t* orp, int32_t* oci, T* ov) {
  const int lane = threadIdx.x & (G - 1);
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) / G; i < n; i += (gridDim.x * blockDim.x) / G) {
    const int o = orp[i], len = orp[i + 1] - o, src = toff ? toff[i] : i * stride;
    for (int t = lane; t < len; t += G) {
      oci[o + t] = tci[src + t];
      ov[o + t] = tv[src + t];
    }
  }
}

template <class T>
void compact_rows(cudaStream_t s, int n, double avg, const int32_t* toff, int stride, const int32_t* tci, const T* tv,
                  DCsr<T>& out) {
  const int G = avg <= 6.0 ? 4 : avg <= 12.0 ? 8 : avg <= 24.0 ? 16 : 32;
  const int cgrid = grid_for((int64_t)n * G, 256);
#define FG_COMPACT(GG)                                                                                            \
  FG_LAUNCH((compact_rows_copy_kernel<T, GG>), cgrid, 256, 0, s, n, toff, stride, tci, tv, out.rp.p, out.ci.p, \
            out.v.p)
  switch (G) {
    case 4: FG_COMPACT(4); break;
    case 8: FG_COMPACT(8); break;
    case 16: FG_COMPACT(16); break;
    default: FG_COMPACT(32); break;
  }
#undef FG_COMPACT
}

// Narrow products whose rows fit this many temporary entries as whole rows (n x ncols) take
// their slots there at once: no count of the products, no scan of the counts and no look at
// their total (two launches and a host read of 10-15 us before a kernel of 10-20 us).
constexpr int64_t kDirectSlots = 1 << 21;

// C = A B.  max_row (or null) receives the longest row of C, read back with its size.  With
// on_device a product that takes direct slots is not read back at all: its arrays have room
// for every slot and C.nnz is that bound (for a product that only the next product reads).
template <class T>
void run_spgemm_hash(Ctx& c, EscArgs<T> a, int nrows_out, int ncols_out, DCsr<T>& out, int* max_row, bool on_device) {
  cudaStream_t s = c.stream;
  PhaseTimer pt(s, -2);
  a.n = nrows_out;
  const size_t dper = dense_warp_smem<T>(ncols_out);
  const bool narrow = nrows_out < 65536 && ncols_out <= kDenseCols;
  DBuf<int32_t> mx(1, s);
  out.n = nrows_out;
  out.m = ncols_out;
  auto dense_rows = [&](const int32_t* toff, int32_t* tci, T* tv, int32_t* cnt) {
    const int wpb = (int)std::max<size_t>(1, std::min<size_t>(8, (size_t)(200 * 1024) / dper));
    const size_t dsm = (size_t)wpb * dper;
    ensure_smem(spgemm_dense_warp_kernel<T>, dsm);
    FG_LAUNCH(spgemm_dense_warp_kernel<T>, (int)std::min<int64_t>((nrows_out + wpb - 1) / wpb, 152 * 4), 32 * wpb,
              dsm, s, a, ncols_out, toff, tci, tv, cnt);
  };
  if (narrow && (int64_t)nrows_out * ncols_out <= kDirectSlots) {
    const int64_t slots = (int64_t)nrows_out * ncols_out;
    DBuf<int32_t> cnt(nrows_out + 1, s), tci(slots, s);
    DBuf<T> tv(slots, s);
    dense_rows(nullptr, tci.p, tv.p, cnt.p);
    pt.mark("sp rows");
    out.rp.alloc(nrows_out + 1, s);
    exclusive_scan_async(cnt.p, out.rp.p, nrows_out, s);
    out.nnz = slots;
    double avg = 16.0;
    if (!on_device) {
      int32_t h_tot = 0, h_max = 0;
      if (max_row) {
        reduce_max_async(cnt.p, nrows_out, mx.p, s);
        FG_CUDA(cudaMemcpyAsync(&h_max, mx.p, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
      }
      FG_CUDA(cudaMemcpyAsync(&h_tot, out.rp.p + nrows_out, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
      FG_CUDA(cudaStreamSynchronize(s));
      g_host_syncs.fetch_add(1, std::memory_order_relaxed);
      out.nnz = h_tot;
      if (max_row) *max_row = h_max;
      avg = nrows_out > 0 ? (double)out.nnz / nrows_out : 0.0;
    }
    out.ci.alloc(out.nnz > 0 ? out.nnz : 1, s);
    out.v.alloc(out.nnz > 0 ? out.nnz : 1, s);
    compact_rows<T>(s, nrows_out, avg, nullptr, ncols_out, tci.p, tv.p, out);
    pt.mark("sp out");
    return;
  }
  DBuf<int32_t> items(nrows_out + 1, s), capv(nrows_out + 1, s), toff(nrows_out + 1, s), cnt(nrows_out + 1, s);
  a.counts = items.p;
  FG_LAUNCH((esc_count_items_kernel<T, ESC_SPGEMM>), grid_for(nrows_out, 256), 256, 0, s, a);
  FG_LAUNCH(spgemm_capacity_kernel, grid_for(nrows_out, 256), 256, 0, s, nrows_out, items.p, ncols_out, capv.p);
  const int64_t tcap = exclusive_scan(capv.p, toff.p, nrows_out, s);
  FG_REQUIRE(tcap < INT32_MAX, FEMGPU_ERR_LIMIT, "SpGEMM temporary exceeds int32 indexing");
  DBuf<int32_t> tci(tcap > 0 ? tcap : 1, s);
  DBuf<T> tv(tcap > 0 ? tcap : 1, s);
  pt.mark("sp items");
  DBuf<int32_t> over1(nrows_out + 1, s), nover1(1, s), over2(nrows_out + 1, s), nover2(1, s);
  nover1.zero();
  nover2.zero();
  const int wgrid = std::min<int64_t>((nrows_out + kHashWarps - 1) / kHashWarps, 152 * 32);
  if (narrow) {
    dense_rows(toff.p, tci.p, tv.p, cnt.p);  // every row on the dense accumulator tier (no overflow rows)
  } else if (nrows_out >= 65536 && tcap <= (int64_t)nrows_out * 128) {
    // short rows on average: thread-per-row tier first, its overflow rows to the warp tier
    DBuf<int32_t> over0(nrows_out + 1, s), nover0(1, s);
    nover0.zero();
    FG_LAUNCH(spgemm_row_kernel<T>, grid_for(nrows_out, kRowThreads), kRowThreads, 0, s, a, toff.p, tci.p, tv.p,
              cnt.p, over0.p, nover0.p);
    FG_LAUNCH(hash_warp_kernel<T>, wgrid, 32 * kHashWarps, 0, s, a, over0.p, nover0.p, toff.p, tci.p, tv.p, cnt.p,
              over1.p, nover1.p);
  } else {
    FG_LAUNCH(hash_warp_kernel<T>, wgrid, 32 * kHashWarps, 0, s, a, (const int32_t*)nullptr,
              (const int32_t*)nullptr, toff.p, tci.p, tv.p, cnt.p, over1.p, nover1.p);
  }
  pt.mark("sp rows");
  // the output offsets are scanned before the overflow count is read, so when no row
  // overflowed (the usual case) both come back in one round trip
  out.rp.alloc(nrows_out + 1, s);
  exclusive_scan_async(cnt.p, out.rp.p, nrows_out, s);
  int32_t h_n1 = 0, h_tot = 0, h_max = 0;
  if (max_row) {
    reduce_max_async(cnt.p, nrows_out, mx.p, s);
    FG_CUDA(cudaMemcpyAsync(&h_max, mx.p, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
  }
  FG_CUDA(cudaMemcpyAsync(&h_n1, nover1.p, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
  FG_CUDA(cudaMemcpyAsync(&h_tot, out.rp.p + nrows_out, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
  FG_CUDA(cudaStreamSynchronize(s));
  g_host_syncs.fetch_add(1, std::memory_order_relaxed);
  const int n1 = h_n1;
  out.nnz = h_tot;
  if (n1 > 0) {
    const size_t bsm = (size_t)kHashBlockCap * (sizeof(unsigned long long) + sizeof(T) + sizeof(int32_t));
    ensure_smem(hash_block_kernel<T>, bsm);
    FG_LAUNCH(hash_block_kernel<T>, std::min(n1, 152 * 2), kHashBlockThreads, bsm, s, a, over1.p, n1, toff.p, tci.p,
              tv.p, cnt.p, over2.p, nover2.p);
    const int n2 = read_scalar(nover2.p, s);
    if (n2 > 0) {
      // more unique columns than the block table: dense accumulator over the columns
      const size_t dsm = (size_t)ncols_out * (sizeof(T) + 1);
      FG_REQUIRE(dsm <= 200 * 1024, FEMGPU_ERR_LIMIT, "SpGEMM row with more than 4096 unique columns");
      EscArgs<T> ad = a;
      ad.nbig = n2;
      ad.big_rows = over2.p;
      ensure_smem(esc_dense_kernel<T, ESC_SPGEMM, false>, dsm);
      ensure_smem(esc_dense_kernel<T, ESC_SPGEMM, true>, dsm);
      ad.counts = cnt.p;
      FG_LAUNCH((esc_dense_kernel<T, ESC_SPGEMM, false>), std::min(n2, 304), 256, dsm, s, ad, ncols_out, nullptr,
                nullptr);
      ad.orp = toff.p;
      ad.oci = tci.p;
      ad.ov = tv.p;
      FG_LAUNCH((esc_dense_kernel<T, ESC_SPGEMM, true>), std::min(n2, 304), 256, dsm, s, ad, ncols_out, nullptr,
                nullptr);
    }
    out.nnz = exclusive_scan(cnt.p, out.rp.p, nrows_out, s);  // the overflow rows' counts are in now
    if (max_row) h_max = reduce_max(cnt.p, nrows_out, s);
  }
  pt.mark("sp big");
  out.ci.alloc(out.nnz > 0 ? out.nnz : 1, s);
  out.v.alloc(out.nnz > 0 ? out.nnz : 1, s);
  if (max_row) *max_row = h_max;
  compact_rows<T>(s, nrows_out, nrows_out > 0 ? (double)out.nnz / nrows_out : 0.0, toff.p, 0, tci.p, tv.p, out);
  pt.mark("sp out");
}

// ---- level matrices -----------------------------------------------------------------
// Diagonal of the sorted rows and its reciprocal.
template <class T>
__global__ void diag_kernel(int n, const int32_t* rp, const int32_t* ci, const T* v, T* d, T* dinv) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    int s = lower_bound_i32(ci, rp[i], rp[i + 1], i);
    const T x = (s < rp[i + 1] && ci[s] == i) ? v[s] : (T)0;
    d[i] = x;
    dinv[i] = (T)1 / x;
  }
}

// In- and out-of-partition entries of every row, and the longest in-partition row in *longest
// (zero before).
template <class T>
__global__ void split_count_kernel(int n, const int32_t* rp, const int32_t* ci, const int32_t* part, int32_t* cin,
                                   int32_t* cout, int32_t* longest) {
  __shared__ int sh[32];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  int a = 0, b = 0;
  if (i < n) {
    const int pi = part[i];
    for (int e = rp[i]; e < rp[i + 1]; e++) {
      const int j = ci[e];
      if (j == i) continue;
      if (part[j] == pi) a++;
      else b++;
    }
    cin[i] = a;
    cout[i] = b;
  }
  const int m = agg_block_max(a, sh);
  if (threadIdx.x == 0 && m > 0) atomicMax(longest, m);
}

template <class T>
__global__ void split_fill_kernel(int n, const int32_t* rp, const int32_t* ci, const T* v, const int32_t* part,
                                  const int32_t* irp, int32_t* ici, T* iv, const int32_t* orp, int32_t* oci, T* ov) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int pi = part[i], qi = irp[i], qo = orp[i];
  for (int e = rp[i]; e < rp[i + 1]; e++) {
    int j = ci[e];
    if (j == i) continue;
    if (part[j] == pi) {
      T val = v[e];
      if (j < i) {  // the symmetric smoother reads the upper entry (j, i) for both
        int u = lower_bound_i32(ci, rp[j], rp[j + 1], i);
        val = (u < rp[j + 1] && ci[u] == i) ? v[u] : (T)0;
      }
      ici[qi] = j;
      iv[qi] = val;
      qi++;
    } else {
      oci[qo] = j;
      ov[qo] = v[e];
      qo++;
    }
  }
}

template <class T>
__global__ void transpose_count_kernel(int64_t nnz, const int32_t* ci, int32_t* cnt) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nnz; e += (int64_t)gridDim.x * blockDim.x)
    atomicAdd(&cnt[ci[e]], 1);
}

template <class T>
__global__ void transpose_fill_kernel(int n, const int32_t* rp, const int32_t* ci, const T* v, const int32_t* trp,
                                      int32_t* cur, int32_t* tci, T* tv) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int e = rp[i]; e < rp[i + 1]; e++) {
    int k = ci[e];
    int q = trp[k] + atomicAdd(&cur[k], 1);
    tci[q] = i;
    tv[q] = v[e];
  }
}

template <class T>
__global__ void cast_kernel(int64_t n, const double* in, T* out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = (T)in[i];
}

template <class T>
__global__ void widen_kernel(int64_t n, const T* __restrict__ in, double* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = (double)in[i];
}

template <class T>
__global__ void narrow_kernel(int64_t n, const double* __restrict__ in, T* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = (T)in[i];
}

template <class T>
__global__ void densify_kernel(int n, const int32_t* rp, const int32_t* ci, const T* v, double* F) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n)
    for (int e = rp[i]; e < rp[i + 1]; e++) F[(int64_t)i * n + ci[e]] = (double)v[e];
}

// Dense LU with partial pivoting (first maximal |pivot| in row order), one block.
__global__ void dense_lu_kernel(int n, double* F, int32_t* piv, int32_t* status) {
  __shared__ double s_best[1024];
  __shared__ int s_idx[1024];
  for (int k = 0; k < n; k++) {
    double best = -1.0;
    int bi = n;
    for (int i = k + threadIdx.x; i < n; i += blockDim.x) {
      double a = fabs(F[(int64_t)i * n + k]);
      if (a > best || (a == best && i < bi)) {
        best = a;
        bi = i;
      }
    }
    s_best[threadIdx.x] = best;
    s_idx[threadIdx.x] = bi;
    __syncthreads();
    for (int off = blockDim.x >> 1; off > 0; off >>= 1) {
      if (threadIdx.x < off) {
        double ob = s_best[threadIdx.x + off];
        int oi = s_idx[threadIdx.x + off];
        if (ob > s_best[threadIdx.x] || (ob == s_best[threadIdx.x] && oi < s_idx[threadIdx.x])) {
          s_best[threadIdx.x] = ob;
          s_idx[threadIdx.x] = oi;
        }
      }
      __syncthreads();
    }
    int p = s_idx[0];
    double pb = s_best[0];
    __syncthreads();
    if (!(pb > 0.0)) {  // every candidate is zero, or NaN (then no row was chosen and p is n)
      if (threadIdx.x == 0) *status = 1;
      return;
    }
    if (threadIdx.x == 0) piv[k] = p;
    if (p != k)
      for (int j = threadIdx.x; j < n; j += blockDim.x) {
        double t = F[(int64_t)k * n + j];
        F[(int64_t)k * n + j] = F[(int64_t)p * n + j];
        F[(int64_t)p * n + j] = t;
      }
    __syncthreads();
    double d = F[(int64_t)k * n + k];
    for (int i = k + 1 + threadIdx.x; i < n; i += blockDim.x) F[(int64_t)i * n + k] = F[(int64_t)i * n + k] / d;
    __syncthreads();
    for (int64_t q = threadIdx.x; q < (int64_t)(n - k - 1) * (n - k - 1); q += blockDim.x) {
      int i = k + 1 + (int)(q / (n - k - 1));
      int j = k + 1 + (int)(q % (n - k - 1));
      F[(int64_t)i * n + j] = fma(-F[(int64_t)i * n + k], F[(int64_t)k * n + j], F[(int64_t)i * n + j]);
    }
    __syncthreads();
  }
}

// The same factorisation on a cluster of kLuCluster CTAs, the matrix in their shared memory
// (n <= kLuMax).  Columns go to the CTAs in panels of kLuPanel (panel p to CTA p mod
// kLuCluster).  Per panel: its CTA factorises it (a thread per row, the row's entries in
// registers) and writes it into every CTA's shared memory; after one cluster barrier each
// CTA applies its row exchanges to its own columns and updates the columns on the right,
// first the panel's rows, then the rows below.  Every entry receives the same
// updates in the same order (k ascending) as in dense_lu_kernel, so the factors keep their
// bits; the matrix is read from CSR and the factors leave column by column, as the inverse
// reads them.  Row exchanges leave as pos[j], the row where the unit entry of e_j ends.
// Bound by the panels' chains (pivot search, division) and by the FP64 pipe: one SM has 2
// FP64 units, so one block spends n^3 / 6 cycles on the updates alone; eight CTAs share
// them.  105 rows: 340 -> 152 us; 2D 64^2: 46 -> 28 us.
constexpr int kLuCluster = 8;
constexpr int kLuPanel = 8;
constexpr int kLuMax = 392;  // the CTA's columns and two panels: 225,792 bytes
constexpr int kLuThreads = 512;

inline size_t lu_smem_bytes(int n) {
  const int panels = (n + kLuPanel - 1) / kLuPanel, own = (panels + kLuCluster - 1) / kLuCluster;
  return (size_t)(own + 2) * kLuPanel * n * sizeof(double);
}

// (key, row) with the largest key, lowest row first, over the warp.
__device__ __forceinline__ void warp_first_max(unsigned long long& key, int& row) {
  const unsigned hi = (unsigned)(key >> 32), mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned lo = hi == mh ? (unsigned)key : 0u, ml = __reduce_max_sync(0xffffffffu, lo);
  const bool top = hi == mh && (unsigned)key == ml;
  row = (int)__reduce_min_sync(0xffffffffu, top ? (unsigned)row : 0xffffffffu);
  key = (unsigned long long)mh << 32 | ml;
}

template <class T>
__global__ void __launch_bounds__(kLuThreads) dense_lu_cluster_kernel(int n, const int32_t* __restrict__ rp,
                                                                      const int32_t* __restrict__ ci,
                                                                      const T* __restrict__ v,
                                                                      double* __restrict__ Fc,
                                                                      int32_t* __restrict__ pos, int32_t* status) {
  extern __shared__ __align__(16) double lu_sm[];
  __shared__ unsigned long long s_key[32];
  __shared__ int s_row[32];
  __shared__ double s_prow[kLuPanel], s_krow[kLuPanel];
  __shared__ int s_piv[kLuMax + kLuPanel];  // every pivot so far
  __shared__ int s_bad;                     // a panel's owner met a zero pivot
  cg::cluster_group cl = cg::this_cluster();
  const int me = (int)cl.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int panels = (n + kLuPanel - 1) / kLuPanel;
  const int own = me < panels ? (panels - me + kLuCluster - 1) / kLuCluster : 0;  // own panels
  double* const cols = lu_sm;  // local column l: rows at cols + l n; l = 8 (panel / 8) + column in panel
  // the current panel, written by its owner; two, so that an owner may write its panel while
  // another CTA still reads the one before
  double* const Lb0 = lu_sm + (size_t)((panels + kLuCluster - 1) / kLuCluster) * kLuPanel * n;
  for (int q = tid; q < own * kLuPanel * n; q += kLuThreads) cols[q] = 0.0;
  if (tid == 0) s_bad = 0;
  cl.sync();  // every CTA is running before another writes its shared memory
  for (int i = warp; i < n; i += kLuThreads / 32)
    for (int e = rp[i] + lane; e < rp[i + 1]; e += 32) {
      const int j = ci[e], p = j / kLuPanel;
      if (p % kLuCluster == me) cols[(size_t)((p / kLuCluster) * kLuPanel + j % kLuPanel) * n + i] = (double)v[e];
    }
  __syncthreads();
  const int nt = (n + 31) / 32 * 32;  // threads of the panel factorisation
  bool bad = false;
  for (int p = 0; p < panels; p++) {
    const int owner = p % kLuCluster, k0 = p * kLuPanel, nk = min(kLuPanel, n - k0);
    double* const Lb = Lb0 + (size_t)(p & 1) * kLuPanel * n;
    if (me == owner && tid < nt) {
      double* const pan = cols + (size_t)(p / kLuCluster) * kLuPanel * n;
      double a[kLuPanel];
#pragma unroll
      for (int c = 0; c < kLuPanel; c++) a[c] = tid < n ? pan[(size_t)c * n + tid] : 0.0;
      bool ok = true;
#pragma unroll
      for (int kk = 0; kk < kLuPanel; kk++) {
        const int k = k0 + kk;
        if (kk < nk && ok) {
          // first maximal |a| at or below the diagonal: magnitudes order like their bits; 0
          // stands for rows above and for NaN, 1 for a zero
          // (integer compares: a floating-point one would take the FP64 pipe)
          unsigned long long key = (unsigned long long)__double_as_longlong(a[kk]) & 0x7fffffffffffffffull;
          key = tid >= k && tid < n && key <= 0x7ff0000000000000ull ? key + 1 : 0;
          int row = tid;
          warp_first_max(key, row);
          if (lane == 0) {
            s_key[warp] = key;
            s_row[warp] = row;
          }
          asm volatile("bar.sync 1, %0;" ::"r"(nt) : "memory");
          key = lane < nt / 32 ? s_key[lane] : 0;
          row = lane < nt / 32 ? s_row[lane] : 0x7fffffff;
          warp_first_max(key, row);
          ok = key > 1;
          if (ok) {
            if (tid == row)
#pragma unroll
              for (int c = 0; c < kLuPanel; c++) s_prow[c] = a[c];
            if (tid == k)
#pragma unroll
              for (int c = 0; c < kLuPanel; c++) s_krow[c] = a[c];
            asm volatile("bar.sync 1, %0;" ::"r"(nt) : "memory");
            double pr[kLuPanel];
#pragma unroll
            for (int c = 0; c < kLuPanel; c++) pr[c] = s_prow[c];
            if (tid == row && row != k)
#pragma unroll
              for (int c = 0; c < kLuPanel; c++) a[c] = s_krow[c];
            if (tid == k)
#pragma unroll
              for (int c = 0; c < kLuPanel; c++) a[c] = pr[c];
            if (tid > k) {
              // a zero (padding rows, sparse columns) keeps its warp out of the division's
              // slow path: +-0 / d is a zero of the product's sign
              const long long ab = __double_as_longlong(a[kk]);
              if ((ab << 1) != 0) a[kk] = a[kk] / pr[kk];
              else a[kk] = __longlong_as_double(ab ^ (__double_as_longlong(pr[kk]) & (1ll << 63)));
#pragma unroll
              for (int c = kk + 1; c < kLuPanel; c++) a[c] = fma(-a[kk], pr[c], a[c]);
            }
            if (tid < kLuCluster) *cl.map_shared_rank(&s_piv[k], tid) = row;
          } else if (tid < kLuCluster) {
            *cl.map_shared_rank(&s_bad, tid) = 1;
          }
        }
      }
      if (tid < n) {
#pragma unroll
        for (int c = 0; c < kLuPanel; c++) pan[(size_t)c * n + tid] = a[c];
        if (tid >= k0)
          for (int d = 0; d < kLuCluster; d++) {
            double* const dst = cl.map_shared_rank(Lb, d);
#pragma unroll
            for (int c = 0; c < kLuPanel; c++) dst[c * n + tid] = a[c];
          }
      }
    }
    cl.sync();  // the panel is everywhere; every CTA is done with the panel before it
    bad = s_bad != 0;
    if (bad) break;
    // own columns outside the panel, eight lanes each: the panel's row exchanges, then (right
    // of the panel) the panel's rows
    const int r = tid & 7;
    for (int l0 = warp * 4; l0 < own * kLuPanel; l0 += kLuThreads / 8) {
      const int l = l0 + (lane >> 3), gp = me + (l / kLuPanel) * kLuCluster;  // global panel
      const bool live = l < own * kLuPanel && gp != p;
      double* const col = cols + (size_t)l * n;
      if (live && r == 0)
        for (int kk = 0; kk < nk; kk++) {
          const int pv = s_piv[k0 + kk];
          if (pv != k0 + kk) {
            const double t = col[k0 + kk];
            col[k0 + kk] = col[pv];
            col[pv] = t;
          }
        }
      __syncwarp();
      const bool right = live && gp > p;
      double x = right && r < nk ? col[k0 + r] : 0.0;
#pragma unroll
      for (int kk = 0; kk < kLuPanel; kk++) {
        const double u = __shfl_sync(0xffffffffu, x, kk, 8);
        if (right && kk < r && r < nk) x = fma(-Lb[kk * n + k0 + r], u, x);
      }
      if (right && r < nk) col[k0 + r] = x;
    }
    __syncthreads();
    // rows below the panel of the own columns right of it (a right column exists only when
    // the panel is full): one warp per column and 32 rows
    const int first = p < me ? 0 : (p - me) / kLuCluster + 1;  // first own panel right of p
    const int ncol = (own - first) * kLuPanel, i0 = k0 + kLuPanel;
    const int chunks = (n - i0 + 31) / 32;
    for (int t = warp; t < ncol * chunks; t += kLuThreads / 32) {
      double* const col = cols + (size_t)(first * kLuPanel + t / chunks) * n;
      const int i = i0 + (t % chunks) * 32 + lane;
      if (i < n) {
        double x = col[i];
#pragma unroll
        for (int kk = 0; kk < kLuPanel; kk++) x = fma(-Lb[kk * n + i], col[k0 + kk], x);
        col[i] = x;
      }
    }
    __syncthreads();
  }
  if (bad) {
    if (me == 0 && tid == 0) *status = 1;
  } else {
    for (int q = tid; q < own * kLuPanel * n; q += kLuThreads) {
      const int l = q / n, j = (me + (l / kLuPanel) * kLuCluster) * kLuPanel + l % kLuPanel;
      if (j < n) Fc[(size_t)j * n + q % n] = cols[q];
    }
    if (me == 0 && tid < n) {
      int at = tid;
      for (int k = 0; k < n; k++) {
        const int pv = s_piv[k];
        at = at == k ? pv : at == pv ? k : at;
      }
      pos[tid] = at;
    }
  }
  cl.sync();  // no CTA leaves while another may still read its shared memory
}

// Column j of the inverse from the factors of dense_lu_cluster_kernel, one warp per column,
// row i in lane i mod 32, register i / 32: the operations of dense_inverse_kernel in the same
// order, with the factors' columns loaded G steps ahead.  Bound by the chain of 2 n steps
// (a shuffle and a fused multiply-add each, and a division in the back substitution).
// 107 rows: 133 -> 101 us.
// Division by d with y = 1 / d at hand (Markstein, "Computation of elementary functions on
// the IBM RISC System/6000 processor", 1990): s y corrected once is within one ulp of s / d,
// its remainder is exact, and a second correction with the correctly rounded reciprocal y
// rounds s / d correctly, unless d's significand is all ones.  That d, and operands whose
// remainders could leave the normal range, take the division itself; a zero s keeps s y.
__device__ __forceinline__ bool recip_usable(double d) {
  const unsigned hi = (unsigned)__double2hiint(d) & 0x7fffffffu, lo = (unsigned)__double2loint(d);
  return hi - 0x20000000u < 0x3fe00000u && !((hi & 0xfffffu) == 0xfffffu && lo == 0xffffffffu);
}
__device__ __forceinline__ double div_by_recip(double s, double d, double y, bool usable) {
  const unsigned hi = (unsigned)__double2hiint(s) & 0x7fffffffu;
  const double q0 = s * y;
  if (usable && hi - 0x20000000u < 0x3fe00000u) {
    const double q1 = fma(fma(-d, q0, s), y, q0);
    return fma(fma(-d, q1, s), y, q1);
  }
  if (usable && (hi | (unsigned)__double2loint(s)) == 0u) return q0;
  return s / d;
}

template <int R, int G>
__global__ void __launch_bounds__(32) dense_inverse_warp_kernel(int n, const double* __restrict__ Fc,
                                                                const int32_t* __restrict__ pos,
                                                                const int32_t* __restrict__ status,
                                                                double* __restrict__ inv) {
  if (*status != 0) return;
  const int j = blockIdx.x, lane = threadIdx.x;
  const int at = pos[j];
  double x[R];
#pragma unroll
  for (int r = 0; r < R; r++) x[r] = lane + 32 * r == at ? 1.0 : 0.0;
  double f[G][R];
  // forward: column q of L, q ascending
#pragma unroll
  for (int r = 0; r < R; r++) {
    auto load = [&](int g, int q) {
#pragma unroll
      for (int s = r; s < R; s++) {
        const int i = lane + 32 * s;
        f[g][s] = (q < n && i < n) ? Fc[(size_t)q * n + i] : 0.0;
      }
    };
#pragma unroll
    for (int g = 0; g < G; g++) load(g, 32 * r + g);
    for (int l0 = 0; l0 < 32 && 32 * r + l0 < n; l0 += G) {
#pragma unroll
      for (int g = 0; g < G; g++) {
        const int q = 32 * r + l0 + g;
        const double b = __shfl_sync(0xffffffffu, x[r], l0 + g);
        if (q < n) {
#pragma unroll
          for (int s = r; s < R; s++)
            if (lane + 32 * s > q) x[s] = fma(-f[g][s], b, x[s]);
        }
        if (l0 + G < 32) load(g, q + G);
      }
    }
  }
  // back: column q of U, q descending; x_q is divided by the diagonal first
  double y[R];  // reciprocals of the diagonal of this lane's rows
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int i = lane + 32 * r;
    y[r] = i < n ? 1.0 / Fc[(size_t)i * n + i] : 1.0;
  }
#pragma unroll
  for (int r = R - 1; r >= 0; r--) {
    auto load = [&](int g, int q) {
#pragma unroll
      for (int s = 0; s <= r; s++) {
        const int i = lane + 32 * s;
        f[g][s] = (q < n && i < n) ? Fc[(size_t)q * n + i] : 1.0;
      }
    };
#pragma unroll
    for (int g = 0; g < G; g++) load(g, 32 * r + 31 - g);
    for (int l0 = 31; l0 >= 0; l0 -= G) {
#pragma unroll
      for (int g = 0; g < G; g++) {
        const int l = l0 - g, q = 32 * r + l;
        if (q < n) {  // the same for the whole warp
          if (lane == l) x[r] = div_by_recip(x[r], f[g][r], y[r], recip_usable(f[g][r]));
          const double b = __shfl_sync(0xffffffffu, x[r], l);
#pragma unroll
          for (int s = r; s >= 0; s--)  // the next step's register first
            if (lane + 32 * s < q) x[s] = fma(-f[g][s], b, x[s]);
        }
        if (l0 - G >= 0) load(g, q - G);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < R; r++)
    if (lane + 32 * r < n) inv[(size_t)(lane + 32 * r) * n + j] = x[r];
}

// Whether dense_inverse takes a coarsest matrix of n rows: it must fit, and the device must be
// able to run the cluster (asked for sizes in steps of 56 rows, one panel more per CTA every
// second step).
template <class T>
bool lu_in_cluster(const Ctx& c, int n) {
  if (n > kLuMax || c.cluster_limit < kLuCluster) return false;
  constexpr int kStep = 56;
  static_assert(kLuMax % kStep == 0, "the largest step is kLuMax");
  const size_t smem = lu_smem_bytes((n + kStep - 1) / kStep * kStep);
  return largest_cluster(reinterpret_cast<const void*>(dense_lu_cluster_kernel<T>), kLuThreads, kLuCluster, smem) ==
         kLuCluster;
}

// The explicit inverse of a coarsest matrix that lu_in_cluster accepts; *status is set when it
// is singular.
template <class T>
void dense_inverse(cudaStream_t s, int n, const int32_t* rp, const int32_t* ci, const T* v, double* F, int32_t* pos,
                   int32_t* status, double* inv) {
  const size_t smem = lu_smem_bytes(n);
  auto lu = dense_lu_cluster_kernel<T>;
  ensure_dynamic_smem(reinterpret_cast<const void*>(lu), smem);  // with the static arrays it may pass 48 KB first
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kLuCluster);
  cfg.blockDim = dim3(kLuThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kLuCluster;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
  FG_CUDA(cudaLaunchKernelEx(&cfg, lu, n, rp, ci, v, F, pos, status));
  auto iv = n <= 64    ? dense_inverse_warp_kernel<2, 8>
            : n <= 128 ? dense_inverse_warp_kernel<4, 8>
            : n <= 256 ? dense_inverse_warp_kernel<8, 4>
                       : dense_inverse_warp_kernel<14, 2>;
  FG_LAUNCH(iv, n, 32, 0, s, n, F, pos, status, inv);
}

// Column j of the inverse (block j): solve L U x = P e_j column by column, so each
// step updates every remaining row in parallel.  Forward: row i takes the updates of
// columns 0, 1, ..., i-1 in that order; back: columns n-1, ..., i+1, then the division
// by U_ii (the CPU oracle uses the same orders).
__global__ void dense_inverse_kernel(int n, const double* __restrict__ F, const int32_t* __restrict__ piv,
                                     double* __restrict__ inv) {
  extern __shared__ double sb[];
  const int j = blockIdx.x;
  for (int i = threadIdx.x; i < n; i += blockDim.x) sb[i] = (i == j) ? 1.0 : 0.0;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int k = 0; k < n; k++) {
      const double t = sb[k];
      sb[k] = sb[piv[k]];
      sb[piv[k]] = t;
    }
  __syncthreads();
  for (int q = 0; q < n; q++) {
    const double bq = sb[q];
    for (int i = q + 1 + threadIdx.x; i < n; i += blockDim.x) sb[i] = fma(-F[(int64_t)i * n + q], bq, sb[i]);
    __syncthreads();
  }
  for (int q = n - 1; q >= 0; q--) {
    if (threadIdx.x == 0) sb[q] = sb[q] / F[(int64_t)q * n + q];
    __syncthreads();
    const double bq = sb[q];
    for (int i = threadIdx.x; i < q; i += blockDim.x) sb[i] = fma(-F[(int64_t)i * n + q], bq, sb[i]);
    __syncthreads();
  }
  for (int i = threadIdx.x; i < n; i += blockDim.x) inv[(int64_t)i * n + j] = sb[i];
}

// First row and first in-partition entry of partitions 0..npart (npart = the end), and the
// largest partition's rows and in-partition entries (mx[0], mx[1]); one block.
__global__ void __launch_bounds__(1024) partition_starts_kernel(int npart, const int32_t* part_idx,
                                                                const int32_t* agg_idx, const int32_t* irp,
                                                                int32_t* row0, int32_t* ent0, int32_t* mx) {
  __shared__ int sh[32];
  int rows = 0, ents = 0;
  for (int p = threadIdx.x; p <= npart; p += 1024) {
    const int r = agg_idx[part_idx[p]], e = irp[r];
    row0[p] = r;
    ent0[p] = e;
    if (p < npart) {
      const int r1 = agg_idx[part_idx[p + 1]];
      rows = max(rows, r1 - r);
      ents = max(ents, irp[r1] - e);
    }
  }
  rows = agg_block_max(rows, sh);
  ents = agg_block_max(ents, sh);
  if (threadIdx.x == 0) {
    mx[0] = rows;
    mx[1] = ents;
  }
}

// Rank of a lane's row in its 32-row block: by decreasing length, ties by row.
__device__ __forceinline__ int block_rank(bool live, int len, int lane) {
  const unsigned key = live ? ((unsigned)(len + 1) << 5) | (unsigned)(31 - lane) : 0u;
  int rank = 0;
  for (int j = 0; j < 32; j++) rank += __shfl_sync(0xffffffffu, key, j) > key;
  return rank;
}

// The copy of x that a lane's column a reads (a < 0: none), the warp's lanes reading together;
// load: per bank, the distinct columns that have chosen it (the warp's scratch).
template <class T, int NC>
__device__ __forceinline__ int choose_copies(int a, int* load) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int NB = sizeof(T) == 4 ? 32 : 16;  // bank slots of one element size
  constexpr int SHIFT = NB / kXCopies;          // bank slots between copies
  if (NC == 1) return 0;
  const int lane = threadIdx.x & 31;
  const unsigned same = __match_any_sync(kAll, a);
  const int leader = __ffs(same) - 1;
  bool choosing = a >= 0 && leader == lane;
  int copy = 0;
  if (lane < NB) load[lane] = 0;
  __syncwarp();
  while (__any_sync(kAll, choosing)) {
    int bank = -1 - lane;
    if (choosing) {
      int best = 0;
#pragma unroll
      for (int c = 0; c < NC; c++) {
        const int lb = load[(a + c * SHIFT) % NB];
        if (c == 0 || lb < best) {
          best = lb;
          copy = c;
        }
      }
      bank = (a + copy * SHIFT) % NB;
    }
    const unsigned rivals = __match_any_sync(kAll, bank);
    __syncwarp();
    if (choosing && __ffs(rivals) - 1 == lane) {
      load[bank]++;
      choosing = false;
    }
    __syncwarp();
  }
  return __shfl_sync(kAll, copy, leader);
}

// The register smoother's entry layout, one CTA of 512 threads per group, warp w taking
// the group's rows [rs + 32w, rs + 32w + 32) (a block):
// * the block's rows are ranked by decreasing in-partition length (ties: lower row
//   first); jrow[block start + p] = offset in the block of the row ranked p;
// * entry k of the row ranked p goes to (block's first entry) + m_0 + ... + m_{k-1} + p,
//   m_j = rows of the block longer than j (a jagged-diagonal layout of the block);
// * each entry's column becomes (column - rs) + c * xcopy_stride<T>(): per diagonal, every
//   distinct column takes the copy c of x whose shared-memory bank holds the fewest distinct
//   columns of that diagonal so far (ties: the lowest copy); equal columns share the first
//   one's copy.  The columns choose in rounds, all at once: of those that want the same bank
//   the lowest lane gets it, the others choose again (4 to 6 rounds; one column after the
//   other took 32 steps: 2.1 M rows 939 -> 546 us, 2,744 rows 45 -> 24 us).
// Entry values and the order of each row's entries are unchanged: only where they sit.
template <class T>
__global__ void __launch_bounds__(512) jds_build_kernel(const int32_t* __restrict__ grows,
                                                        const int32_t* __restrict__ irp,
                                                        const int32_t* __restrict__ ici, const T* __restrict__ iv,
                                                        T* __restrict__ jv, uint16_t* __restrict__ jc,
                                                        uint8_t* __restrict__ jrow) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int CS = xcopy_stride<T>();
  constexpr int NB = sizeof(T) == 4 ? 32 : 16;  // bank slots of one element size
  const int rs = grows[blockIdx.x], re = grows[blockIdx.x + 1];
  const int lane = threadIdx.x & 31;
  const int r0 = rs + (threadIdx.x & ~31);
  if (r0 >= re) return;  // the whole warp: its block is empty
  const int row = r0 + lane;
  const bool live = row < re;
  const int len = live ? irp[row + 1] - irp[row] : 0;
  const int rank = block_rank(live, len, lane);
  if (live) jrow[r0 + rank] = (uint8_t)lane;
  const int eb = irp[r0];
  const int mine = live ? irp[row] : 0;
  __shared__ int s_load[16][NB];  // per warp and bank: distinct columns of this diagonal
  int* const load = s_load[threadIdx.x >> 5];
  int dk = 0;  // entries on the diagonals before k
  for (int k = 0;; k++) {
    const bool act = k < len;
    const unsigned am = __ballot_sync(kAll, act);
    if (!am) break;
    const int a = act ? ici[mine + k] - rs : -1;
    const int copy = choose_copies<T, kXCopies>(a, load);
    if (act) {
      const int dst = eb + dk + rank;
      jv[dst] = iv[mine + k];
      jc[dst] = (uint16_t)(a + copy * CS);
    }
    dk += __popc(am);
  }
}

// Padded row lengths of the row smoother's layout: whole quads.
__global__ void quad_len_kernel(int n, const int32_t* __restrict__ irp, int32_t* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = (irp[i + 1] - irp[i] + 3) & ~3;
}

// The row smoother's entry layout: blocks, ranks and copies as in jds_build_kernel, but four
// consecutive entries of a row stay together (one 128-bit load of FP32 values, one 64-bit load
// of columns).  Quad q of the row ranked p starts at qrp[block's first row] + 4 (m_0 + ... +
// m_{q-1} + p), m_q = rows of the block longer than 4 q; a row's last quad is filled with zero
// values that point at the zero slot kRegGroupRows of copy 0.  qrp: exclusive scan of
// quad_len_kernel's lengths.
template <class T, int NC>
__global__ void __launch_bounds__(512) quad_build_kernel(const int32_t* __restrict__ grows,
                                                         const int32_t* __restrict__ irp,
                                                         const int32_t* __restrict__ ici, const T* __restrict__ iv,
                                                         const int32_t* __restrict__ qrp, T* __restrict__ rv,
                                                         uint16_t* __restrict__ rc, uint8_t* __restrict__ rrow) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int CS = xcopy_stride<T>();
  const int rs = grows[blockIdx.x], re = grows[blockIdx.x + 1];
  const int lane = threadIdx.x & 31;
  const int r0 = rs + (threadIdx.x & ~31);
  if (r0 >= re) return;  // the whole warp: its block is empty
  const int row = r0 + lane;
  const bool live = row < re;
  const int mine = live ? irp[row] : 0;
  const int len = live ? irp[row + 1] - mine : 0;
  const int rank = block_rank(live, len, lane);
  if (live) rrow[r0 + rank] = (uint8_t)lane;
  __shared__ int s_load[16][sizeof(T) == 4 ? 32 : 16];
  int* const load = s_load[threadIdx.x >> 5];
  int at = qrp[r0] + 4 * rank;
  for (int q = 0;; q += 4) {
    const unsigned am = __ballot_sync(kAll, q < len);
    if (!am) break;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const bool act = q + i < len;
      const int a = act ? ici[mine + q + i] - rs : -1;
      const int copy = choose_copies<T, NC>(a, load);
      if (q < len) {
        rv[at + i] = act ? iv[mine + q + i] : (T)0;
        rc[at + i] = (uint16_t)(act ? a + copy * CS : kRegGroupRows);
      }
    }
    at += 4 * __popc(am);
  }
}

// Smoother work groups: consecutive partitions packed greedily into one CTA while
// the group stays within `max_rows` rows and `max_ents` in-partition entries.
// hr, he: first row and first in-partition entry of partitions 0..npart.
template <class T>
void build_smoother_groups(Ctx& c, Level<T>& L, int max_rows, int max_ents, const std::vector<int32_t>& hr,
                           const std::vector<int32_t>& he) {
  cudaStream_t s = c.stream;
  std::vector<int32_t> g{hr[0]};
  int gp = 0, mx = 0, mxe = 0;
  for (int p = 1; p <= L.npart; p++) {
    const bool last = p == L.npart;
    if (last || hr[p + 1] - hr[gp] > max_rows || he[p + 1] - he[gp] > max_ents) {
      g.push_back(hr[p]);
      mx = std::max(mx, hr[p] - hr[gp]);
      mxe = std::max(mxe, he[p] - he[gp]);
      gp = p;
    }
  }
  L.ngroups = (int)g.size() - 1;
  L.max_group_rows = mx;
  L.max_group_ents = mxe;
  L.grows.alloc(g.size(), s);
  L.grows.upload(g.data(), g.size());
}

// ci[e] = map[ci[e]]
__global__ void map_columns_kernel(int64_t nnz, const int32_t* __restrict__ map, int32_t* ci) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e < nnz) ci[e] = map[ci[e]];
}

// len[i] = length of row src[i] of rp
__global__ void gather_row_lengths_kernel(int m, const int32_t* __restrict__ src, const int32_t* __restrict__ rp,
                                          int32_t* __restrict__ len) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < m) len[i] = rp[src[i] + 1] - rp[src[i]];
}

// Row i of the output is row src[i] of the input (one warp per row, entries in order).
template <class T>
__global__ void gather_rows_kernel(int m, const int32_t* __restrict__ src, const int32_t* __restrict__ rp,
                                   const int32_t* __restrict__ ci, const T* __restrict__ v,
                                   const int32_t* __restrict__ orp, int32_t* __restrict__ oci, T* __restrict__ ov) {
  const int i = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (i >= m) return;
  const int a = rp[src[i]], len = rp[src[i] + 1] - a, o = orp[i];
  for (int t = lane; t < len; t += 32) {
    oci[o + t] = ci[a + t];
    ov[o + t] = v[a + t];
  }
}

template <class T>
void build_levels(Ctx& c, Hierarchy<T>& H) {
  cudaStream_t s = c.stream;
  const int n0 = c.A.n;
  // level 0: the operator converted to T
  {
    auto L0 = std::make_unique<Level<T>>();
    L0->n = n0;
    L0->A.n = L0->A.m = n0;
    L0->A.nnz = c.A.nnz;
    L0->A.rp.alloc(n0 + 1, s);
    L0->A.ci.alloc(c.A.nnz, s);
    L0->A.v.alloc(c.A.nnz, s);
    FG_CUDA(cudaMemcpyAsync(L0->A.rp.p, c.A.rp.p, (n0 + 1) * sizeof(int32_t), cudaMemcpyDeviceToDevice, s));
    FG_CUDA(cudaMemcpyAsync(L0->A.ci.p, c.A.ci.p, c.A.nnz * sizeof(int32_t), cudaMemcpyDeviceToDevice, s));
    FG_LAUNCH(cast_kernel<T>, grid_for(c.A.nnz, 256), 256, 0, s, c.A.nnz, c.A.v.p, L0->A.v.p);
    L0->gnnz = c.graph_nnz;
    L0->max_row = c.A_max_row;
    L0->gxadj.alloc(n0 + 1, s);
    L0->gadj.alloc(c.graph_nnz > 0 ? c.graph_nnz : 1, s);
    FG_CUDA(cudaMemcpyAsync(L0->gxadj.p, c.gxadj.p, (n0 + 1) * sizeof(int32_t), cudaMemcpyDeviceToDevice, s));
    if (c.graph_nnz > 0)
      FG_CUDA(cudaMemcpyAsync(L0->gadj.p, c.gadj.p, c.graph_nnz * sizeof(int32_t), cudaMemcpyDeviceToDevice, s));
    H.L.push_back(std::move(L0));
  }
  int num_levels = 1;
  while (true) {
    Level<T>& L = *H.L.back();
    const int N = L.A.n;
    if (N < c.cfg.topSize || num_levels >= c.cfg.maxLevels) {
      FG_REQUIRE(N <= 8192, FEMGPU_ERR_LIMIT, "coarsest level too large for the dense solve (raise maxLevels)");
      L.coarsest = true;
      DBuf<double> F((size_t)N * N, s);
      DBuf<int32_t> piv(N, s), st(1, s);
      st.zero();
      L.Ainv.alloc((size_t)N * N, s);
      if (L.A64v.n ? lu_in_cluster<double>(c, N) : lu_in_cluster<T>(c, N)) {
        if (L.A64v.n)  // formed in FP64: the dense factorisation takes those values
          dense_inverse<double>(s, N, L.A.rp.p, L.A.ci.p, L.A64v.p, F.p, piv.p, st.p, L.Ainv.p);
        else
          dense_inverse<T>(s, N, L.A.rp.p, L.A.ci.p, L.A.v.p, F.p, piv.p, st.p, L.Ainv.p);
        FG_REQUIRE(read_scalar(st.p, s) == 0, FEMGPU_ERR_BREAKDOWN, "coarsest matrix is singular");
      } else {
        F.zero();
        if (L.A64v.n)
          FG_LAUNCH(densify_kernel<double>, grid_for(N, 128), 128, 0, s, N, L.A.rp.p, L.A.ci.p, L.A64v.p, F.p);
        else
          FG_LAUNCH(densify_kernel<T>, grid_for(N, 128), 128, 0, s, N, L.A.rp.p, L.A.ci.p, L.A.v.p, F.p);
        FG_LAUNCH(dense_lu_kernel, 1, 1024, 0, s, N, F.p, piv.p, st.p);
        FG_REQUIRE(read_scalar(st.p, s) == 0, FEMGPU_ERR_BREAKDOWN, "coarsest matrix is singular");
        const size_t bbytes = (size_t)N * sizeof(double);
        ensure_smem(dense_inverse_kernel, bbytes);
        FG_LAUNCH(dense_inverse_kernel, N, std::min(1024, std::max(32, (N + 31) / 32 * 32)), bbytes, s, N, F.p, piv.p,
                  L.Ainv.p);
      }
      L.b.alloc(N, s);
      L.x.alloc(N, s);
      break;
    }
    PhaseTimer pt(s, num_levels - 1);
    const TraceRange level_range("femgpu setup: level");
    OldMisOut o;
    old_mis(c, N, L.gnnz, L.gxadj.p, L.gadj.p, o);
    pt.mark("aggregate");
    L.nagg = o.nagg;
    L.npart = o.npart;
    L.perm = std::move(o.perm);
    L.iperm = std::move(o.iperm);
    L.agg_idx = std::move(o.agg_idx);
    L.part_idx = std::move(o.part_idx);
    L.agg_of = std::move(o.agg_of);
    // permuted operator
    {
      EscArgs<T> a{};
      a.arp = L.A.rp.p;
      a.aci = L.A.ci.p;
      a.av = L.A.v.p;
      a.perm = L.perm.p;
      a.iperm = L.iperm.p;
      a.known_nnz = L.A.nnz;
      a.max_items = L.max_row;
      run_esc_sort<T, ESC_PERMUTE>(c, a, N, N, L.Ap);
    }
    pt.mark("permute");
    L.diag.alloc(N, s);
    L.dinv.alloc(N, s);
    FG_LAUNCH(diag_kernel<T>, grid_for(N, 256), 256, 0, s, N, L.Ap.rp.p, L.Ap.ci.p, L.Ap.v.p, L.diag.p, L.dinv.p);
    // in/out-of-partition split; the two entry counts, the three maxima and the partition
    // starts the smoother plan needs come back in one round trip
    std::vector<int32_t> hr, he;
    {
      DBuf<int32_t> cin(N + 1, s), cout(N + 1, s), row0(L.npart + 1, s), ent0(L.npart + 1, s), mx(3, s);
      mx.zero();
      FG_LAUNCH(split_count_kernel<T>, grid_for(N, 256), 256, 0, s, N, L.Ap.rp.p, L.Ap.ci.p, o.part_of_row.p, cin.p,
                cout.p, mx.p + 2);
      L.Ain.n = L.Ain.m = L.Aout.n = L.Aout.m = N;
      L.Ain.rp.alloc(N + 1, s);
      L.Aout.rp.alloc(N + 1, s);
      exclusive_scan_async(cin.p, L.Ain.rp.p, N, s);
      exclusive_scan_async(cout.p, L.Aout.rp.p, N, s);
      FG_LAUNCH(partition_starts_kernel, 1, 1024, 0, s, L.npart, L.part_idx.p, L.agg_idx.p, L.Ain.rp.p, row0.p,
                ent0.p, mx.p);
      int32_t h_in = 0, h_out = 0, h_mx[3] = {0, 0, 0};
      hr.resize(L.npart + 1);
      he.resize(L.npart + 1);
      FG_CUDA(cudaMemcpyAsync(&h_in, L.Ain.rp.p + N, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
      FG_CUDA(cudaMemcpyAsync(&h_out, L.Aout.rp.p + N, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
      FG_CUDA(cudaMemcpyAsync(h_mx, mx.p, 3 * sizeof(int32_t), cudaMemcpyDeviceToHost, s));
      row0.download(hr.data(), L.npart + 1);
      ent0.download(he.data(), L.npart + 1);
      FG_CUDA(cudaStreamSynchronize(s));
      g_host_syncs.fetch_add(1, std::memory_order_relaxed);
      L.Ain.nnz = h_in;
      L.Aout.nnz = h_out;
      L.max_part_rows = h_mx[0];
      L.max_part_entries = h_mx[1];
      L.max_in_row = h_mx[2];
      L.Ain.ci.alloc(L.Ain.nnz > 0 ? L.Ain.nnz : 1, s);
      L.Ain.v.alloc(L.Ain.nnz + 16, s);  // slack for 16-byte rounded bulk copies
      L.Ain.v.zero();
      L.Aout.ci.alloc(L.Aout.nnz > 0 ? L.Aout.nnz : 1, s);
      L.Aout.v.alloc(L.Aout.nnz > 0 ? L.Aout.nnz : 1, s);
      FG_LAUNCH(split_fill_kernel<T>, grid_for(N, 256), 256, 0, s, N, L.Ap.rp.p, L.Ap.ci.p, L.Ap.v.p,
                o.part_of_row.p, L.Ain.rp.p, L.Ain.ci.p, L.Ain.v.p, L.Aout.rp.p, L.Aout.ci.p, L.Aout.v.p);
    }
    {
      pt.mark("split rows");
      if (smoother_in_registers(L.max_in_row, L.max_part_rows)) {
        build_smoother_groups(c, L, kRegGroupRows, std::numeric_limits<int>::max(), hr, he);
        L.jv.alloc(L.Ain.nnz + 16, s);
        L.jv.zero();
        L.jc16.alloc(L.Ain.nnz + 16, s);
        L.jc16.zero();
        L.jrow.alloc(N, s);
        if (L.ngroups > 0)
          FG_LAUNCH(jds_build_kernel<T>, L.ngroups, kRegGroupRows, 0, s, L.grows.p, L.Ain.rp.p, L.Ain.ci.p,
                    L.Ain.v.p, L.jv.p, L.jc16.p, L.jrow.p);
      } else
        build_smoother_groups(c, L, L.max_part_rows, L.max_part_entries, hr, he);
      pt.mark("groups");
      plan_smoother(c, L);
      pt.mark("plan");
      if (pt.on)
        fprintf(stderr,
                "[femgpu setup] level %d smoother: %s, groups %d (max %d rows), lanes %d, cluster %d, "
                "slice %d rows / %d entries, %d threads, %zu B shared%s\n",
                num_levels - 1,
                smoother_in_registers(L.max_in_row, L.max_part_rows) ? "registers"
                : L.rows_c > 0                                        ? "rows"
                : L.smooth_k > 0                                      ? "cluster, entries in registers"
                                                                      : "cluster",
                L.ngroups, L.max_group_rows, L.smooth_lanes, L.cluster, L.slice_rows, L.slice_ents,
                L.smooth_threads, L.smooth_smem, L.smooth_staged ? ", staged" : "");
    }
    pt.mark("split");
    // prolongator and restrictor
    {
      EscArgs<T> a{};
      a.arp = L.Ap.rp.p;
      a.aci = L.Ap.ci.p;
      a.av = L.Ap.v.p;
      a.agg_of = L.agg_of.p;
      a.diag = L.diag.p;
      a.neg_omega = -(T)c.cfg.proOmega;
      a.max_items = L.max_row > 0 ? L.max_row + 1 : 0;
      run_esc_sort<T, ESC_PROLONG>(c, a, N, L.nagg, L.P);
    }
    {
      pt.mark("P");
      DCsr<T> Ru;  // unsorted transpose, then rows sorted by column
      Ru.n = L.nagg;
      Ru.m = N;
      Ru.nnz = L.P.nnz;
      DBuf<int32_t> cnt(L.nagg + 1, s), cur(L.nagg, s);
      cnt.zero();
      cur.zero();
      FG_LAUNCH(transpose_count_kernel<T>, grid_for(L.P.nnz, 256), 256, 0, s, L.P.nnz, L.P.ci.p, cnt.p);
      Ru.rp.alloc(L.nagg + 1, s);
      exclusive_scan_async(cnt.p, Ru.rp.p, L.nagg, s);
      Ru.ci.alloc(L.P.nnz, s);
      Ru.v.alloc(L.P.nnz, s);
      FG_LAUNCH(transpose_fill_kernel<T>, grid_for(N, 256), 256, 0, s, N, L.P.rp.p, L.P.ci.p, L.P.v.p, Ru.rp.p, cur.p,
                Ru.ci.p, Ru.v.p);
      EscArgs<T> a{};
      a.arp = Ru.rp.p;
      a.aci = Ru.ci.p;
      a.av = Ru.v.p;
      a.known_nnz = L.P.nnz;
      a.max_items = N <= kEscWarpCap ? N : 0;  // a row of R has at most N entries
      run_esc_sort<T, ESC_PERMUTE>(c, a, L.nagg, N, L.R);
    }
    // Galerkin product A_next = R (Ap P)
    auto nx = std::make_unique<Level<T>>();
    if (sizeof(T) == 4 && (int64_t)L.nagg <= (int64_t)kFp64GalerkinPerTop * c.cfg.topSize) {
      // the coarse end of a mixed hierarchy: the product in FP64 on widened operands
      DBuf<double> apv(L.Ap.nnz > 0 ? L.Ap.nnz : 1, s), pv(L.P.nnz > 0 ? L.P.nnz : 1, s),
          rv(L.R.nnz > 0 ? L.R.nnz : 1, s);
      FG_LAUNCH(widen_kernel<T>, grid_for(L.Ap.nnz, 256), 256, 0, s, L.Ap.nnz, L.Ap.v.p, apv.p);
      FG_LAUNCH(widen_kernel<T>, grid_for(L.P.nnz, 256), 256, 0, s, L.P.nnz, L.P.v.p, pv.p);
      FG_LAUNCH(widen_kernel<T>, grid_for(L.R.nnz, 256), 256, 0, s, L.R.nnz, L.R.v.p, rv.p);
      DCsr<double> AP, A64;
      EscArgs<double> a{};
      a.arp = L.Ap.rp.p;
      a.aci = L.Ap.ci.p;
      a.av = apv.p;
      a.brp = L.P.rp.p;
      a.bci = L.P.ci.p;
      a.bv = pv.p;
      run_spgemm_hash<double>(c, a, N, L.nagg, AP, nullptr, true);
      EscArgs<double> r{};
      r.arp = L.R.rp.p;
      r.aci = L.R.ci.p;
      r.av = rv.p;
      r.brp = AP.rp.p;
      r.bci = AP.ci.p;
      r.bv = AP.v.p;
      run_spgemm_hash<double>(c, r, L.nagg, L.nagg, A64, &nx->max_row, false);
      nx->A.n = A64.n;
      nx->A.m = A64.m;
      nx->A.nnz = A64.nnz;
      nx->A.rp = std::move(A64.rp);
      nx->A.ci = std::move(A64.ci);
      nx->A.v.alloc(A64.nnz > 0 ? A64.nnz : 1, s);
      FG_LAUNCH(narrow_kernel<T>, grid_for(A64.nnz, 256), 256, 0, s, A64.nnz, A64.v.p, nx->A.v.p);
      nx->A64v = std::move(A64.v);
      pt.mark("RAP");
    } else {
      DCsr<T> AP;
      EscArgs<T> a{};
      a.arp = L.Ap.rp.p;
      a.aci = L.Ap.ci.p;
      a.av = L.Ap.v.p;
      a.brp = L.P.rp.p;
      a.bci = L.P.ci.p;
      a.bv = L.P.v.p;
      pt.mark("R");
      run_spgemm_hash<T>(c, a, N, L.nagg, AP, nullptr, true);
      pt.mark("AP");
      EscArgs<T> r{};
      r.arp = L.R.rp.p;
      r.aci = L.R.ci.p;
      r.av = L.R.v.p;
      r.brp = AP.rp.p;
      r.bci = AP.ci.p;
      r.bv = AP.v.p;
      run_spgemm_hash<T>(c, r, L.nagg, L.nagg, nx->A, &nx->max_row, false);
      pt.mark("RAP");
    }
    nx->n = L.nagg;
    nx->gxadj = std::move(o.xadj_out);
    nx->gadj = std::move(o.adj_out);
    nx->gnnz = o.nnz_out;
    // work vectors
    L.b.alloc(N, s);
    L.x.alloc(N, s);
    L.r.alloc(N, s);
    L.xo.alloc(N, s);
    L.t.alloc(N, s);
    L.bp.alloc(N, s);
    autotune_level(c, L);  // result-neutral launch choices, timed on this level's data
    H.L.push_back(std::move(nx));
    num_levels++;
  }
  H.num_levels = num_levels;
  // The V-cycle keeps every non-coarsest level's vectors in that level's own (permuted)
  // order: each parent's restriction writes its rows in the child's order and its
  // prolongation reads the child's vector by the child's new indices, so no separate
  // permutation runs per cycle.  Entry order within each row is kept (same sums).
  for (size_t l = 0; l + 1 < H.L.size(); l++) {
    Level<T>& L = *H.L[l];
    const Level<T>& N = *H.L[l + 1];
    if (L.coarsest || N.coarsest) continue;
    if (L.P.nnz > 0)
      FG_LAUNCH(map_columns_kernel, grid_for(L.P.nnz, 256), 256, 0, s, L.P.nnz, N.perm.p, L.P.ci.p);
    const int m = L.R.n;
    DCsr<T> Rp;
    Rp.n = m;
    Rp.m = L.R.m;
    Rp.nnz = L.R.nnz;
    DBuf<int32_t> len(m + 1, s);
    Rp.rp.alloc(m + 1, s);
    FG_LAUNCH(gather_row_lengths_kernel, grid_for(m, 256), 256, 0, s, m, N.iperm.p, L.R.rp.p, len.p);
    exclusive_scan_async(len.p, Rp.rp.p, m, s);
    Rp.ci.alloc(L.R.nnz > 0 ? L.R.nnz : 1, s);
    Rp.v.alloc(L.R.nnz > 0 ? L.R.nnz : 1, s);
    FG_LAUNCH(gather_rows_kernel<T>, grid_for((int64_t)m * 32, 256), 256, 0, s, m, N.iperm.p, L.R.rp.p, L.R.ci.p,
              L.R.v.p, Rp.rp.p, Rp.ci.p, Rp.v.p);
    L.R = std::move(Rp);
  }
}

__global__ void identity_kernel(int n, int32_t* p) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = i;
}

}  // namespace

std::atomic<int64_t> g_kernel_launches{0};
std::atomic<int64_t> g_host_syncs{0};
thread_local cudaMemPool_t g_alloc_pool = nullptr;
thread_local BlockCache* g_alloc_cache = nullptr;

// Values of perm(A) on its (sorted) pattern: row i' and column j' of the permuted
// matrix are row iperm[i'] and column iperm[j'] of A, found by binary search.
__global__ void permuted_values_kernel(int n, const int32_t* __restrict__ prp, const int32_t* __restrict__ pci,
                                       const int32_t* __restrict__ iperm, const int32_t* __restrict__ arp,
                                       const int32_t* __restrict__ aci, const double* __restrict__ av,
                                       double* __restrict__ pv) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int r = iperm[i], a0 = arp[r], a1 = arp[r + 1];
  for (int e = prp[i]; e < prp[i + 1]; e++) {
    const int q = lower_bound_i32(aci, a0, a1, iperm[pci[e]]);
    pv[e] = av[q];
  }
}

// Entries of each 32-row slice (32 x its longest row), for the sliced layout of the
// permuted FP64 operator.
__global__ void slice_width_kernel(int n, int nslices, const int32_t* __restrict__ prp, int32_t* __restrict__ cnt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if ((i >> 5) >= nslices) return;  // whole warps: nslices * 32 threads are live
  const int len = i < n ? prp[i + 1] - prp[i] : 0;
  const int w = __reduce_max_sync(0xffffffffu, len);
  if ((i & 31) == 0) cnt[i >> 5] = 32 * w;
}

// The permuted operator written as slices: row i's entry k (in the sorted pattern's
// order) goes to off[i / 32] + 32 k + i % 32, its value looked up in A as in
// permuted_values_kernel; the slice's remaining slots get column -1 and value 0.
__global__ void sliced_values_kernel(int n, int nslices, const int32_t* __restrict__ prp,
                                     const int32_t* __restrict__ pci, const int32_t* __restrict__ iperm,
                                     const int32_t* __restrict__ arp, const int32_t* __restrict__ aci,
                                     const double* __restrict__ av, const int32_t* __restrict__ off,
                                     int32_t* __restrict__ sci, double* __restrict__ sv) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int sl = i >> 5;
  if (sl >= nslices) return;
  const int base = off[sl] + (i & 31), w = (off[sl + 1] - off[sl]) >> 5;
  int k = 0;
  if (i < n) {
    const int r = iperm[i], a0 = arp[r], a1 = arp[r + 1], e0 = prp[i], e1 = prp[i + 1];
    for (; k < e1 - e0; k++) {
      const int col = pci[e0 + k];
      sci[base + 32 * k] = col;
      sv[base + 32 * k] = av[lower_bound_i32(aci, a0, a1, iperm[col])];
    }
  }
  for (; k < w; k++) {
    sci[base + 32 * k] = -1;
    sv[base + 32 * k] = 0.0;
  }
}

void amg_setup(Ctx& c) {
  cudaStream_t s = c.stream;
  FG_REQUIRE(c.has_matrix, FEMGPU_ERR_NOT_READY,
             "no operator: call femgpu_set_mesh + femgpu_assemble or femgpu_set_matrix_csr");
  FG_REQUIRE(c.cfg.aggregatorType == 0, FEMGPU_ERR_INVALID, "only aggregatorType 0 (OldMIS) is implemented");
  cudaEvent_t e0, e1;
  FG_CUDA(cudaEventCreate(&e0));
  FG_CUDA(cudaEventCreate(&e1));
  FG_CUDA(cudaEventRecord(e0, s));
  c.H.reset();
  c.has_hierarchy = false;
  const int n = c.A.n;
  const int32_t* perm0 = nullptr;
  if (c.cfg.precision == 1) {
    auto H = std::make_unique<Hierarchy<double>>();
    build_levels(c, *H);
    if (!H->L[0]->coarsest) perm0 = H->L[0]->perm.p;
    c.H = std::move(H);
  } else {
    auto H = std::make_unique<Hierarchy<float>>();
    build_levels(c, *H);
    if (!H->L[0]->coarsest) perm0 = H->L[0]->perm.p;
    c.H = std::move(H);
  }
  c.perm0.alloc(n, s);
  if (perm0)
    FG_CUDA(cudaMemcpyAsync(c.perm0.p, perm0, n * sizeof(int32_t), cudaMemcpyDeviceToDevice, s));
  else
    FG_LAUNCH(identity_kernel, grid_for(n, 256), 256, 0, s, n, c.perm0.p);
  // FP64 outer operator in level-0 order: the pattern of the level-0 permuted operator
  // (already built, rows sorted by column), values looked up in the FP64 matrix
  {
    DBuf<int32_t> iperm(n, s);
    FG_LAUNCH(invert_kernel, grid_for(n, 256), 256, 0, s, n, c.perm0.p, iperm.p);
    const int32_t *prp, *pci;
    int64_t pnnz;
    if (c.cfg.precision == 1) {
      const Level<double>& L0 = *static_cast<Hierarchy<double>&>(*c.H).L[0];
      prp = L0.coarsest ? c.A.rp.p : L0.Ap.rp.p;
      pci = L0.coarsest ? c.A.ci.p : L0.Ap.ci.p;
      pnnz = L0.coarsest ? c.A.nnz : L0.Ap.nnz;
    } else {
      const Level<float>& L0 = *static_cast<Hierarchy<float>&>(*c.H).L[0];
      prp = L0.coarsest ? c.A.rp.p : L0.Ap.rp.p;
      pci = L0.coarsest ? c.A.ci.p : L0.Ap.ci.p;
      pnnz = L0.coarsest ? c.A.nnz : L0.Ap.nnz;
    }
    c.A0p.n = c.A0p.m = n;
    c.A0p.nnz = pnnz;
    c.A0p.rp.alloc(n + 1, s);
    FG_CUDA(cudaMemcpyAsync(c.A0p.rp.p, prp, (n + 1) * sizeof(int32_t), cudaMemcpyDeviceToDevice, s));
    // Slices of 32 rows when they pad the operator by at most 1/8 (mesh operators,
    // whose neighbouring rows have similar lengths); otherwise CSR.
    const int nslices = (n + 31) / 32;
    c.sliced = false;
    c.s_off.release();
    c.s_ci.release();
    c.s_v.release();
    c.A0p.ci.release();
    c.A0p.v.release();
    if (n > 0) {
      c.s_off.alloc(nslices + 1, s);
      FG_LAUNCH(slice_width_kernel, grid_for((int64_t)nslices * 32, 256), 256, 0, s, n, nslices, c.A0p.rp.p,
                c.s_off.p);
      const int64_t padded = exclusive_scan(c.s_off.p, c.s_off.p, nslices, s);
      if (padded <= INT32_MAX && padded <= pnnz + pnnz / 8) {
        c.sliced = true;
        c.s_padded = padded;
        c.s_ci.alloc(padded > 0 ? padded : 1, s);
        c.s_v.alloc(padded > 0 ? padded : 1, s);
        FG_LAUNCH(sliced_values_kernel, grid_for((int64_t)nslices * 32, 128), 128, 0, s, n, nslices, c.A0p.rp.p,
                  pci, iperm.p, c.A.rp.p, c.A.ci.p, c.A.v.p, c.s_off.p, c.s_ci.p, c.s_v.p);
      } else {
        c.s_off.release();
      }
    }
    if (!c.sliced) {
      c.A0p.ci.alloc(pnnz > 0 ? pnnz : 1, s);
      c.A0p.v.alloc(pnnz > 0 ? pnnz : 1, s);
      if (pnnz > 0)
        FG_CUDA(cudaMemcpyAsync(c.A0p.ci.p, pci, pnnz * sizeof(int32_t), cudaMemcpyDeviceToDevice, s));
      FG_LAUNCH(permuted_values_kernel, grid_for(n, 128), 128, 0, s, n, c.A0p.rp.p, c.A0p.ci.p, iperm.p, c.A.rp.p,
                c.A.ci.p, c.A.v.p, c.A0p.v.p);
    }
  }
  FG_CUDA(cudaEventRecord(e1, s));
  FG_CUDA(cudaEventSynchronize(e1));
  float ms = 0;
  FG_CUDA(cudaEventElapsedTime(&ms, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  c.setup_ms = ms;
  c.has_hierarchy = true;
  c.hier_gen++;  // invalidates the captured PCG iteration graph
}

// The row smoother's layout of a level (quad_build_kernel), with the copies of x spread over the
// banks or (copies == 1) the plain columns.
template <class T>
void build_row_layout(Ctx& c, Level<T>& L, int copies) {
  cudaStream_t s = c.stream;
  const size_t cap = (size_t)L.Ain.nnz + 3 * (size_t)L.n + 16;  // padded rows, slack for bulk copies
  L.rv.alloc(cap, s);
  L.rc.alloc(cap, s);
  L.rrow.alloc(L.n, s);
  L.qrp.alloc((size_t)L.n + 1, s);
  DBuf<int32_t> len(L.n, s);
  FG_LAUNCH(quad_len_kernel, grid_for(L.n, 256), 256, 0, s, L.n, L.Ain.rp.p, len.p);
  exclusive_scan_async(len.p, L.qrp.p, L.n, s);
  auto k = copies == 1 ? quad_build_kernel<T, 1> : quad_build_kernel<T, kXCopies>;
  FG_LAUNCH(k, L.ngroups, kRegGroupRows, 0, s, L.grows.p, L.Ain.rp.p, L.Ain.ci.p, L.Ain.v.p, L.qrp.p, L.rv.p, L.rc.p,
            L.rrow.p);
}
template void build_row_layout<float>(Ctx&, Level<float>&, int);
template void build_row_layout<double>(Ctx&, Level<double>&, int);

}  // namespace femgpu
