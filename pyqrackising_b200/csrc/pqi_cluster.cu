// libpqi: steepest single-flip ascent of one state spread over a thread-block
// cluster (distributed shared memory), for low latency per flip on large n.
//
// A cluster of C CTAs runs one task (graph, starting state) at a time. CTA r
// owns nodes [r*S, r*S + S) (S = n / C rounded up to 32, so every 32-node bit
// word belongs to one CTA). Each thread owns NG groups of four nodes,
// lo + 4*(t + T*j) + i, and keeps their local fields y = W x and their bits in
// registers for the whole ascent.
//
// Per flip:
//   1. every thread applies the previous flip k to its fields
//      (y_v += coef * W_kv, one float4 / char4 of row k per group; the owner of
//      k toggles its bit) and folds the new gains g_v = x_v y_v into a local
//      argmax: float gain first, then the lowest node (a 64-bit key);
//      (branch-free; with it and a row prefetch only for candidates that change,
//      n = 6000 int8, 20 tasks on clusters of 8, went from 4.47 to 3.61 ms and
//      n = 8192 float, 8 tasks, from 6.98 to 6.06, 5.37 with the loads of kAhead);
//   2. warp maxima (two 32-bit redux steps) meet in shared memory behind the
//      flip's one CTA barrier; warp 0 reduces them and its lanes 0..C-1 write the
//      CTA's best (key, exact gain) into slot [rank] of every CTA with st.async,
//      which counts the bytes on that CTA's mbarrier;
//   3. every warp waits (bounded) for the C slots of the flip and reduces them
//      itself to the same global best, flipped next if its gain is > 0. (Warps
//      that each sent to every CTA, with no barrier, took 1.2 times as long.)
// Two slot arrays and two mbarriers alternate between flips; a CTA sends flip
// f + 2 only after every CTA has sent f + 1, so all its warps have read f, and a
// slot array is never rewritten while read. The selection rule is the batched
// kernel's (pqi_batch_search), so both give the same trajectory. Control flow
// depends only on values every warp reads identically, with one exception: a wait
// that runs out does so for one warp (or lane) at a time. It raises the CTA's flag
// of this exchange and the warp goes on with what its slots hold - older keys of
// this task, or 0 - so it stays within the graph. Every warp passes exactly one CTA
// barrier after an exchange, the next flip's or, if it saw no flip left, the one
// behind the loop, and reads the flag behind it: the CTA leaves together. (Flags
// alternate, so that none is raised while a slow warp has yet to read the one
// before.) The other CTAs, which it no longer sends to, follow by their own waits;
// the cluster's barriers stand outside the loop, the same number for every CTA. So
// the flip budget and the bounded waits end every loop. (It costs 1.6 % of a float
// flip: n = 8192, 8 tasks on clusters of 8 5.37 -> 5.46 ms, and none of an int8 one;
// with the verdict in the maximum, or by a reducing barrier, 4 to 8 %.)
#include <cooperative_groups.h>

#include <algorithm>
#include <type_traits>

#include "pqi_common.cuh"
#include "pqi_tc.cuh"

namespace cg = cooperative_groups;

namespace pqi {

// Starting fields of the dense-graph tasks (pqi_batch.cu), freed by the caller.
pqi_status start_fields(const void* graphs, const int* task_graph, const uint32_t* init_states,
                        int words_pitch, int tasks, int max_n, bool i8, cudaStream_t s,
                        double** out, int* pitch);

struct ClusterGraph {  // same layout as the batched search's graph descriptor
  const void* W;
  int n;
  int ld;
  int kind;
  int pad;
  double upper_sum;
  const void* adj_ptr;  // row lists (unused here)
  const void* adj_col;
  const void* adj_val;
};

struct Slot {
  unsigned long long key;  // ord(float gain) << 32 | (0x3FFFFFFF - node) << 1 | bit
  double g;                // exact gain of that node
};

constexpr int kMaxCluster = 16;
constexpr int kMaxWarps = 8;  // per CTA

// In place of rank 0's best when the target is reached: above every key, and its
// gain (a NaN) not above 0.
constexpr unsigned long long kStopKey = ~0ull;

__device__ __forceinline__ unsigned long long flip_key(float gv, int u, int xu) {
  return ((unsigned long long)ord_f32(gv) << 32) |
         (unsigned long long)(((0x3FFFFFFFu - (uint32_t)u) << 1) | (uint32_t)xu);
}

__device__ __forceinline__ int key_node(unsigned long long key) {
  return (int)(0x3FFFFFFFu - (((uint32_t)key) >> 1));
}

__device__ __forceinline__ float key_gain(unsigned long long key) {
  return unord_f32((uint32_t)(key >> 32));
}

// max of a 64-bit key over the warp: two 32-bit reductions (high word, then the
// low word among the lanes holding the highest high word)
__device__ __forceinline__ unsigned long long warp_max_key(unsigned long long key) {
  const uint32_t hi = __reduce_max_sync(0xFFFFFFFFu, (uint32_t)(key >> 32));
  const uint32_t lo =
      __reduce_max_sync(0xFFFFFFFFu, ((uint32_t)(key >> 32) == hi) ? (uint32_t)key : 0u);
  return ((unsigned long long)hi << 32) | lo;
}

// The thread's groups of row k (slice from node lo; group j at lo + 4 (t + T j)).
// Volatile, so that the loads ahead of their use are issued where they stand.
template <typename WT, int NG>
__device__ __forceinline__ void load_row(const WT* __restrict__ row, int v0, int step, int n, WT (&w)[4 * NG]) {
#pragma unroll
  for (int j = 0; j < NG; ++j) {
    const int v = v0 + step * j;
#pragma unroll
    for (int i = 0; i < 4; ++i) w[4 * j + i] = (WT)0;
    if (v < n) {  // (rows are zero padded to a multiple of 128)
      if constexpr (sizeof(WT) == 4) {
        asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(w[4 * j]), "=f"(w[4 * j + 1]), "=f"(w[4 * j + 2]), "=f"(w[4 * j + 3])
                     : "l"(row + v));
      } else {
        uint32_t q;
        asm volatile("ld.global.nc.b32 %0, [%1];" : "=r"(q) : "l"(row + v));
#pragma unroll
        for (int i = 0; i < 4; ++i) w[4 * j + i] = (WT)(int8_t)(q >> (8 * i));
      }
    }
  }
}

// CTAS is the register budget (CTAs of 256 threads per SM): the host takes the
// larger one unless the smaller saves passes over the resident clusters.
// Loads ahead of the choice pay for float slices of one group per thread on the
// larger budget only: n = 8192, 8 tasks on clusters of 8 6.06 -> 5.37 ms, 32 tasks
// 7.23 -> 6.77; int8 rows (n = 6000, 20 tasks) 3.61 -> 4.09, many resident clusters
// (n = 8192, 100 tasks, clusters of 16) 16.2 -> 19.7.
template <typename WT, int NG, int CTAS>
constexpr bool kAhead = sizeof(WT) == 4 && NG == 1 && CTAS == 2;

template <typename WT, int NG, int CTAS>
__global__ void __launch_bounds__(256, CTAS) cluster_ascent_kernel(
    const ClusterGraph* __restrict__ graphs, const int* __restrict__ task_graph,
    const uint32_t* __restrict__ init_states, int words_pitch, int tasks, int spin,
    int flip_budget, uint32_t* __restrict__ best_states, double* __restrict__ best_values,
    unsigned long long* __restrict__ flips_total, int* __restrict__ status, double target,
    int* __restrict__ reached, const double* __restrict__ start_fields, int fields_pitch) {
  typedef typename std::conditional<sizeof(WT) == 1, int, double>::type GT;
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks();
  const int rank = (int)cl.block_rank();
  extern __shared__ __align__(16) unsigned char smem[];
  // slots[p][r]: CTA r's best of the flips with parity p, written here by CTA r
  __shared__ __align__(16) Slot slots[2][kMaxCluster];
  __shared__ unsigned long long red_key[kMaxWarps];
  __shared__ __align__(8) uint64_t bar[2];
  __shared__ double qslot[kMaxCluster];
  __shared__ double red_g[kMaxWarps];
  __shared__ int abort_flag;
  __shared__ int wait_failed[2];  // by parity of the exchange
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int T = blockDim.x, nwarps = T >> 5;
  if (threadIdx.x == 0) {
    tc::mbar_init(&bar[0], 1);
    tc::mbar_init(&bar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    abort_flag = 0;
    wait_failed[0] = wait_failed[1] = 0;
  }
  cl.sync();
  // lane r's view of CTA r: this CTA's slot and the barrier of even exchanges
  uint32_t rslot = 0, rbar = 0;
  if (lane < C) {
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rslot) : "r"(tc::smem_u32(&slots[0][rank])), "r"(lane));
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rbar) : "r"(tc::smem_u32(&bar[0])), "r"(lane));
  }
  uint32_t seq = 0;  // exchanges so far (over all tasks)
  const int clusters = gridDim.x / C;
  for (int task = blockIdx.x / C; task < tasks; task += clusters) {
    const ClusterGraph G = graphs[task_graph[task]];
    const int n = G.n, n32 = (n + 31) >> 5;
    const WT* __restrict__ W = static_cast<const WT*>(G.W);
    const int S = (((n + C - 1) / C) + 31) & ~31;
    const int lo = rank * S, hi = min(n, lo + S);
    uint32_t* bits = reinterpret_cast<uint32_t*>(smem);
    GT* y0 = reinterpret_cast<GT*>(smem + (((size_t)n32 * 4 + 15) & ~size_t(15)));
    for (int w = threadIdx.x; w < n32; w += T) bits[w] = init_states[(size_t)task * words_pitch + w];
    __syncthreads();
    // starting local fields of the slice: computed beforehand for all tasks
    // (start_fields_kernel), else one warp per row
    if (start_fields && !G.adj_ptr) {
      const double* __restrict__ yrow = start_fields + (size_t)task * fields_pitch;
      for (int v = lo + (int)threadIdx.x; v < hi; v += T) y0[v - lo] = (GT)yrow[v];
    } else {
      for (int v = lo + warp; v < hi; v += nwarps) {
        const WT* row = W + (size_t)v * G.ld;
        GT acc = 0;
        for (int u = lane; u < n; u += 32) {
          const GT w = (GT)row[u];
          acc += ((bits[u >> 5] >> (u & 31)) & 1) ? w : -w;
        }
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, o);
        if (lane == 0) y0[v - lo] = acc;
      }
    }
    __syncthreads();
    GT y[4 * NG];
    uint32_t xm = 0;  // bit 4j+i: the bit of node lo + 4*(t + T*j) + i
    double qp = 0.0;
#pragma unroll
    for (int j = 0; j < NG; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int v = lo + 4 * ((int)threadIdx.x + T * j) + i;
        y[4 * j + i] = 0;
        if (v < hi) {
          y[4 * j + i] = y0[v - lo];
          const uint32_t b = (bits[v >> 5] >> (v & 31)) & 1;
          xm |= b << (4 * j + i);
          qp += b ? (double)y[4 * j + i] : -(double)y[4 * j + i];
        }
      }
    // q = sum_v x_v y_v over the cluster: partials stored into every CTA and
    // summed in rank order (the same double everywhere)
    for (int o = 16; o > 0; o >>= 1) qp += __shfl_xor_sync(0xFFFFFFFFu, qp, o);
    if (lane == 0) red_g[warp] = qp;
    __syncthreads();
    if ((int)threadIdx.x < C) {
      double a = 0.0;
      for (int i = 0; i < nwarps; ++i) a += red_g[i];
      *cl.map_shared_rank(&qslot[rank], (int)threadIdx.x) = a;
    }
    // (no key of another task: a warp whose wait runs out goes on with what is there)
    if (threadIdx.x < 2 * kMaxCluster) slots[threadIdx.x & 1][threadIdx.x >> 1].key = 0ull;
    cl.sync();
    double q = 0.0;
    for (int r = 0; r < C; ++r) q += qslot[r];
    const double scale = spin ? 2.0 : 1.0;
    double val = spin ? -q / 2.0 : (2.0 * G.upper_sum - q) / 4.0;
    unsigned long long nflips = 0;
    int timeout = 0, failed = 0;
    int k = -1;
    GT coef = 0;
    // the two runners-up of the last exchange, their row groups in flight
    constexpr bool SPEC = kAhead<WT, NG, CTAS>;
    const int vt = lo + 4 * (int)threadIdx.x;
    int p1 = -1, p2 = -1, ahead = -1;
    WT w1[4 * NG], w2[4 * NG];
    unsigned long long sk = 0ull, gkey = 0ull;  // the last exchange: my lane's slot, the best
    double gk = 0.0;
    for (int f = 0;; ++f) {
      if (k >= 0) {
        // apply the previous flip (node k) to my fields
        WT w[4 * NG];
        if (SPEC && k == p1) {
#pragma unroll
          for (int e = 0; e < 4 * NG; ++e) w[e] = w1[e];
        } else if (SPEC && k == p2) {
#pragma unroll
          for (int e = 0; e < 4 * NG; ++e) w[e] = w2[e];
        } else {
          load_row<WT, NG>(W + (size_t)k * G.ld, vt, 4 * T, n, w);
        }
#pragma unroll
        for (int j = 0; j < 4 * NG; ++j) y[j] += coef * (GT)w[j];
        const int rel = k - lo;
        if (rel >= 0 && rel < S) {
          const int grp = rel >> 2;
          if (grp % T == (int)threadIdx.x) xm ^= 1u << (4 * (grp / T) + (rel & 3));
        }
      }
      // target mode: a task whose value reaches the target raises the global
      // flag; every 16 flips rank 0 reads it and sends kStopKey as its best, so
      // all CTAs stop at the same flip (fields and bits then hold every accepted
      // flip)
      int stop = 0;
      if (reached && (f & 15) == 15 && rank == 0 && threadIdx.x == 0) {
        if (val >= target) atomicExch(reached, 1);
        stop = *(volatile int*)reached;
      }
      // my best flip: float gain first, then the lowest node (nodes ascend)
      float bv = -INFINITY;
      GT bg = 0;
      int be = -1;  // element << 1 | bit
#pragma unroll
      for (int e = 0; e < 4 * NG; ++e) {
        const uint32_t xv = (xm >> e) & 1u;
        GT g;
        if constexpr (sizeof(WT) == 4) {
          g = __hiloint2double(__double2hiint(y[e]) ^ (int)(xv ? 0u : 0x80000000u), __double2loint(y[e]));
        } else {
          g = xv ? y[e] : -y[e];
        }
        const float gv = (float)g;
        const bool up = vt + 4 * T * (e >> 2) + (e & 3) < hi && gv > bv;  // strict: the lowest node keeps a tie
        bv = up ? gv : bv;
        bg = up ? g : bg;
        be = up ? (int)(2 * e + xv) : be;
      }
      const unsigned long long key =
          be >= 0 ? flip_key(bv, vt + 4 * T * (be >> 3) + ((be >> 1) & 3), be & 1) : 0ull;
      const unsigned long long wkey = warp_max_key(key);
      if (lane == 0) red_key[warp] = wkey;
      if (key != 0ull && key == wkey) red_g[warp] = (double)bg;
      const uint32_t par = seq & 1u, ph = (seq >> 1) & 1u;
      ++seq;
      if (threadIdx.x == 0) tc::mbar_expect_tx(&bar[par], (uint32_t)(C * sizeof(Slot)));
      __syncthreads();
      failed = wait_failed[par ^ 1];  // another warp's last wait ran out
      if (warp == 0) {
        // this CTA's best into slot [rank] of every CTA, counted on its bar[par]
        const unsigned long long ck = lane < nwarps ? red_key[lane] : 0ull;
        const double cgv = lane < nwarps ? red_g[lane] : 0.0;
        unsigned long long cb = warp_max_key(ck);
        const uint32_t src = __ballot_sync(0xFFFFFFFFu, ck == cb);
        const double cbg = __shfl_sync(0xFFFFFFFFu, cgv, __ffs(src) - 1);
        // the next row is one of the C CTAs' candidates: pull this CTA's
        // candidate row into L2 while the exchange is in flight (a hint only;
        // a row is ld * sizeof(WT) bytes, 16-byte aligned, inside W)
        if (lane == 0 && cb != 0ull && key_gain(cb) > 0.0f && key_node(cb) != ahead) {
          ahead = key_node(cb);  // (one that stays the best is there already)
          const WT* cand = W + (size_t)ahead * G.ld;
          asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(cand),
                       "r"((uint32_t)((size_t)G.ld * sizeof(WT)))
                       : "memory");
        }
        if (reached && __shfl_sync(0xFFFFFFFFu, stop, 0)) cb = kStopKey;
        if (lane < C) {
          asm volatile(
              "st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.u64 [%0], {%1, %2}, [%3];" ::"r"(
                  rslot + par * (uint32_t)sizeof(slots[0])),
              "l"(cb), "l"(__double_as_longlong(cbg)), "r"(rbar + par * 8u)
              : "memory");
        }
      }
      // While the exchange is in flight: the rows of the last exchange's second
      // and third best, one of which is the next flip in half of the cases
      // (measured on a dense Gaussian graph of 8192 nodes: 0.36 and 0.18).
      if constexpr (SPEC) {
        const unsigned long long s1 = sk == gkey ? 0ull : sk, k1 = warp_max_key(s1);
        const unsigned long long k2 = warp_max_key(s1 == k1 ? 0ull : s1);
        p1 = p2 = -1;
        if (k1 != 0ull) {
          p1 = key_node(k1);
          load_row<WT, NG>(W + (size_t)p1 * G.ld, vt, 4 * T, n, w1);
        }
        if (k2 != 0ull) {
          p2 = key_node(k2);
          load_row<WT, NG>(W + (size_t)p2 * G.ld, vt, 4 * T, n, w2);
        }
      }
      if (failed) break;
      if (!tc::mbar_wait_spin(&bar[par], ph)) wait_failed[par] = 1;
      // the cluster's best (identical in every warp whose wait succeeded)
      sk = lane < C ? slots[par][lane].key : 0ull;
      const double sg = lane < C ? slots[par][lane].g : 0.0;
      gkey = warp_max_key(sk);
      if (rank == 0 && warp == 0) {  // the value is kept by warp 0 of CTA 0
        const uint32_t gsrc = __ballot_sync(0xFFFFFFFFu, sk == gkey);
        gk = __shfl_sync(0xFFFFFFFFu, sg, __ffs(gsrc) - 1);
      }
      const bool none = gkey == 0ull || !(key_gain(gkey) > 0.0f);
      if (none || f >= flip_budget) {
        timeout = !none;
        __syncthreads();  // (the one that warps which go on pass in their next flip)
        failed = wait_failed[par];
        break;
      }
      k = key_node(gkey);
      coef = (gkey & 1ull) ? (GT)-2 : (GT)2;
      val += scale * gk;
      ++nflips;
    }
    if (reached && rank == 0 && threadIdx.x == 0 && val >= target) atomicExch(reached, 1);
    // (the last accepted flip was applied by the pass that found no further one)
    // bits back to shared memory: eight lanes assemble one 32-node word
#pragma unroll
    for (int j = 0; j < NG; ++j) {
      const int v0 = lo + 4 * ((int)threadIdx.x + T * j);
      uint32_t wd = ((xm >> (4 * j)) & 15u) << (4 * (lane & 7));
      wd |= __shfl_xor_sync(0xFFFFFFFFu, wd, 1);
      wd |= __shfl_xor_sync(0xFFFFFFFFu, wd, 2);
      wd |= __shfl_xor_sync(0xFFFFFFFFu, wd, 4);
      if ((lane & 7) == 0 && v0 < hi) bits[v0 >> 5] = wd;
    }
    if (failed && threadIdx.x == 0) *cl.map_shared_rank(&abort_flag, 0) = 1;
    cl.sync();  // all slices final before rank 0 gathers the bits
    if (rank == 0) {
      for (int w = threadIdx.x; w < n32; w += T)
        best_states[(size_t)task * words_pitch + w] = *cl.map_shared_rank(&bits[w], (w * 32) / S);
      if (threadIdx.x == 0) {
        best_values[task] = val;
        atomicAdd(flips_total, nflips);
        if (timeout) atomicExch(status, PQI_ETIMEOUT);
      }
    }
    const int stop = *cl.map_shared_rank(&abort_flag, 0);
    cl.sync();  // no CTA starts the next task while another still reads its bits
    if (stop) {
      // a peer stopped answering: report and leave (every CTA read the flag)
      if (rank == 0 && threadIdx.x == 0) atomicExch(status, PQI_ETIMEOUT);
      return;
    }
  }
}

}  // namespace pqi

using namespace pqi;

extern "C" pqi_status pqi_cluster_ascent(const void* graphs, int num_graphs,
                                         const int* task_graph, const uint32_t* init_states,
                                         int words_pitch, int tasks, int max_n, int kind,
                                         int is_spin_glass, int cluster_size, int flip_budget,
                                         uint32_t* best_states, double* best_values,
                                         unsigned long long* flips_total, int* status,
                                         double target, int* reached, void* stream) {
  PQI_CHECK_ARG(graphs && num_graphs > 0 && task_graph && init_states && tasks > 0 && max_n > 0);
  PQI_CHECK_ARG(best_states && best_values && flips_total && status && flip_budget > 0);
  PQI_CHECK_ARG(cluster_size == 2 || cluster_size == 4 || cluster_size == 8 ||
                cluster_size == 16);
  PQI_CHECK_ARG(words_pitch >= (max_n + 31) / 32);
  PQI_CHECK_ARG(max_n < (1 << 30));
  const bool i8 = kind == PQI_W_I8;
  const int S = (((max_n + cluster_size - 1) / cluster_size) + 31) & ~31;
  // threads: one group of four nodes each where the slice allows, up to 256;
  // groups per thread (held in registers) rounded up to a power of two
  const int groups = (S + 3) / 4;
  const int T = std::max(32, std::min(256, (groups + 31) / 32 * 32));
  int NG = (groups + T - 1) / T;
  NG = NG <= 1 ? 1 : NG <= 2 ? 2 : NG <= 4 ? 4 : NG <= 8 ? 8 : 0;
  if (NG == 0) {
    set_error_text("cluster ascent: graph too large for this cluster size (use 16)");
    return PQI_EINVAL;
  }
  const size_t smem = (((size_t)((max_n + 31) >> 5) * 4 + 15) & ~size_t(15)) +
                      (size_t)S * (i8 ? sizeof(int) : sizeof(double));
  if (smem > 200 * 1024) {
    set_error_text("cluster ascent: slice does not fit in shared memory");
    return PQI_EINVAL;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(T);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = as_stream(stream);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster_size;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const ClusterGraph* gd = static_cast<const ClusterGraph*>(graphs);
  // the starting fields of dense-graph tasks, one pass over W per task tile
  double* sf = nullptr;
  int sf_pitch = 0;
  {
    pqi_status r = start_fields(graphs, task_graph, init_states, words_pitch, tasks, max_n, i8,
                                as_stream(stream), &sf, &sf_pitch);
    if (r != PQI_OK) return r;
  }
  // clusters resident at once (the occupancy query is cached per kernel and
  // launch shape: it is slow on first use)
  auto resident = [&](auto kern, int* out) -> pqi_status {
    PQI_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    if (cluster_size > 8)
      PQI_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    struct FitEntry {
      const void* k;
      size_t smem;
      int T, cs, dev, fit;
    };
    static thread_local FitEntry cache[32];
    static thread_local int cached = 0;
    int dev = 0;
    PQI_TRY(cudaGetDevice(&dev));
    int fit = 0;
    for (int e = 0; e < cached; ++e)
      if (cache[e].k == (const void*)kern && cache[e].smem == smem && cache[e].T == T &&
          cache[e].cs == cluster_size && cache[e].dev == dev)
        fit = cache[e].fit;
    if (fit == 0) {
      cfg.gridDim = dim3(cluster_size);
      PQI_TRY(cudaOccupancyMaxActiveClusters(&fit, kern, &cfg));
      if (fit > 0 && cached < 32) cache[cached++] = {(const void*)kern, smem, T, cluster_size, dev, fit};
    }
    if (fit < 1) {
      set_error_text("cluster ascent: the cluster does not fit on the device");
      return PQI_EINVAL;
    }
    *out = fit;
    return PQI_OK;
  };
  // Two register budgets: a flip takes up to 12 % longer with the smaller one
  // (n = 8192, clusters of 8), so it is for task counts where more resident
  // clusters save passes over them (32 tasks on clusters of 16: 10.1 -> 7.0 ms).
  auto launch = [&](auto fast, auto lean) -> pqi_status {
    int ff = 0, fl = 0;
    pqi_status r = resident(fast, &ff);
    if (r == PQI_OK) r = resident(lean, &fl);
    if (r != PQI_OK) return r;
    const long long wf = (tasks + ff - 1) / ff, wl = (tasks + fl - 1) / fl;
    const auto kern = wl * 9 < wf * 8 ? lean : fast;
    cfg.gridDim = dim3(std::max(1, std::min(tasks, kern == lean ? fl : ff)) * cluster_size);
    PQI_TRY(cudaLaunchKernelEx(&cfg, kern, gd, task_graph, init_states, words_pitch, tasks,
                               is_spin_glass, flip_budget, best_states, best_values, flips_total,
                               status, target, reached, (const double*)sf, sf_pitch));
    return PQI_OK;
  };
  auto pick = [&](auto wt) -> pqi_status {
    using WT = decltype(wt);
    return NG == 1   ? launch(cluster_ascent_kernel<WT, 1, 2>, cluster_ascent_kernel<WT, 1, 4>)
           : NG == 2 ? launch(cluster_ascent_kernel<WT, 2, 2>, cluster_ascent_kernel<WT, 2, 3>)
           : NG == 4 ? launch(cluster_ascent_kernel<WT, 4, 1>, cluster_ascent_kernel<WT, 4, 2>)
                     : launch(cluster_ascent_kernel<WT, 8, 1>, cluster_ascent_kernel<WT, 8, 1>);
  };
  const pqi_status st = i8 ? pick(int8_t{}) : pick(float{});
  if (st != PQI_OK) return st;
  PQI_LAUNCHED("cluster_ascent_kernel");
  if (sf) PQI_TRY(cudaFreeAsync(sf, as_stream(stream)));
  return PQI_OK;
}
