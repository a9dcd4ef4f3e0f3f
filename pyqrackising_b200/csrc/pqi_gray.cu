// libpqi: parallel Gray-code search (replaces the reference's `gray` kernel,
// pyqrackising/kernels.cl:894-978) and the device-resident single-flip
// descent (the repeated single-flip passes of spin_glass_solver.py:605-627).
//
// Both keep each state's gain vector on chip and update it in O(n) per
// accepted flip (g_v -= 2 x_v x_k W_kv, g_k = -g_k) instead of recomputing an
// O(n) row sum for every candidate flip as the reference does.
#include <cooperative_groups.h>

#include <algorithm>
#include <type_traits>

#include "pqi_common.cuh"
#include "pqi_tc.cuh"

namespace pqi {

// Gain storage: exact int32 for int8 weights, float64 otherwise.
template <typename WT>
struct GainOf {
  typedef double type;
};
template <>
struct GainOf<int8_t> {
  typedef int type;
};

__device__ __forceinline__ int bit_of(const uint64_t* bits, int v) {
  return (int)((bits[v >> 6] >> (v & 63)) & 1ull);
}

template <typename GT>
__device__ __forceinline__ GT from_f64(double v);
template <>
__device__ __forceinline__ double from_f64<double>(double v) {
  return v;
}
template <>
__device__ __forceinline__ int from_f64<int>(double v) {
  return (int)llrint(v);
}

// One CTA per seed (grid-stride). Dynamic smem: 64-bit state words, one 32-bit
// word per 64-node block of which of its first 32 nodes have a gain > 0, then
// the gains (unless g_global is given: then CTA b uses g_global + b*n).
//
// The walk visits iterations i = s + m S < iters_bound in order and in each the
// nodes ctz(i + 1) + 64 b, b ascending, and flips those with a gain > 0 (i + 1
// < 2^31, so only the first 31 nodes of a block are ever visited). Flips are
// few from a local optimum, so the walk does not test position by position:
// between flips the set of positive gains is fixed, and an iteration can be
// passed over when no block has a positive node of its class c = ctz(i + 1).
// `any` is the OR of the blocks' words; a warp tests 32 iterations per step
// against it, then finds the block within the first that has one. Every flip
// refreshes the words by ballot as it updates the gains. All warps walk alike
// (identical ballots), so only flips need barriers. Times: see pqi_gray.
constexpr int kGrayThreads = 512;

template <typename WT>
__global__ void __launch_bounds__(kGrayThreads) gray_kernel(
    const WT* __restrict__ Wp, int ld, int n, const uint64_t* __restrict__ theta64,
    const double* __restrict__ base_g, int spin, long long iters_bound, int S,
    uint64_t* __restrict__ theta_out, float* __restrict__ energy_out,
    typename GainOf<WT>::type* g_global) {
  typedef typename GainOf<WT>::type GT;
  extern __shared__ __align__(16) unsigned char smem[];
  const int blocks = (n + 63) >> 6;
  uint64_t* bits = reinterpret_cast<uint64_t*>(smem);
  uint32_t* pos = reinterpret_cast<uint32_t*>(bits + blocks);
  GT* g = g_global ? g_global + (size_t)blockIdx.x * n
                   : reinterpret_cast<GT*>(smem + (((size_t)blocks * 12 + 15) & ~size_t(15)));
  const int lane = threadIdx.x & 31;

  // Flip node k: every thread updates its gains and the words of positive
  // gains, then one thread toggles the bit (read again only after the next
  // flip's first barrier). Reached by all threads with the same k.
  auto flip = [&](int k) {
    __syncthreads();  // every warp has read the gains and words of its choice; the last toggle is done
    const int xk = bit_of(bits, k);
    const WT* __restrict__ row = Wp + (size_t)k * ld;
    constexpr int CH = 16;  // loads in flight per thread
    for (int base = threadIdx.x; base < 64 * blocks; base += CH * kGrayThreads) {
      WT w[CH];
#pragma unroll
      for (int i = 0; i < CH; ++i) {
        const int v = base + i * kGrayThreads;
        w[i] = v < n ? __ldg(row + v) : (WT)0;
      }
#pragma unroll
      for (int i = 0; i < CH; ++i) {
        const int v = base + i * kGrayThreads;
        if (v - lane >= 64 * blocks) break;  // (the warp's 32 nodes are past the last block)
        bool up = false;
        if (v < n) {
          GT y = g[v];
          if (v == k) {
            y = -y;
          } else {
            const GT w2 = (GT)2 * (GT)w[i];
            y += (bit_of(bits, v) == xk) ? -w2 : w2;
          }
          g[v] = y;
          up = y > (GT)0;
        }
        const unsigned m = __ballot_sync(0xFFFFFFFFu, up);
        if (lane == 0 && !(v & 32)) pos[v >> 6] = m;
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) bits[k >> 6] ^= 1ull << (k & 63);
  };

  for (int s = blockIdx.x; s < S; s += gridDim.x) {
    for (int q = threadIdx.x; q < blocks; q += blockDim.x) bits[q] = theta64[q];
    for (int v = threadIdx.x; v < 64 * blocks; v += blockDim.x) {
      const GT y = v < n ? from_f64<GT>(base_g[v]) : (GT)0;
      if (v < n) g[v] = y;
      const unsigned m = __ballot_sync(0xFFFFFFFFu, v < n && y > (GT)0);
      if (lane == 0 && !(v & 32)) pos[v >> 6] = m;
    }
    __syncthreads();

    // Seed mask of work-item s (kernels.cl:915-926): seed bit 63-b flips node
    // n-1-b through a 32-bit int shift, so the mask is 1 << (offset & 31),
    // sign-extended to 64 bits when the count is 31. Every thread computes it.
    const uint64_t seed = (uint64_t)s ^ ((uint64_t)s >> 1);
    const int w0 = (n > 64 ? n - 64 : 0) >> 6;
    uint64_t m[2] = {0ull, 0ull};
    const int max_lcv = n < 64 ? n : 64;
    for (int b = 0; b < max_lcv; ++b) {
      if (!((seed >> (63 - b)) & 1ull)) continue;
      const int off = n - (b + 1);
      const int32_t m32 = (int32_t)(1u << ((unsigned)off & 31u));
      m[(off >> 6) - w0] ^= (uint64_t)(int64_t)m32;
    }
    // Apply the mask one node at a time; the sum of the successive gains is
    // the prologue's cut change (kernels.cl:928-941).
    double E = 0.0;
    for (int q = 0; q < 2; ++q) {
      uint64_t mq = m[q];
      while (mq) {
        const int p = __ffsll((long long)mq) - 1;
        mq &= mq - 1;
        const int node = ((w0 + q) << 6) + p;
        if (node < n) {
          E += (double)g[node];
          flip(node);
        } else if (node < (blocks << 6)) {
          // padding bit of the last word: no energy, kept for the output words
          __syncthreads();
          if (threadIdx.x == 0) bits[node >> 6] ^= 1ull << (node & 63);
        }
      }
    }

    auto any_class = [&]() {
      uint32_t a = 0;
      for (int b = lane; b < blocks; b += 32) a |= pos[b];
      return __reduce_or_sync(0xFFFFFFFFu, a);
    };
    const long long Pm = iters_bound > s ? (iters_bound - 1 - s) / S + 1 : 0;
    long long mi = 0;  // iteration, and its first block still to visit
    int b0 = 0;
    uint32_t any = any_class();
    while (mi < Pm) {
      const long long mm = mi + lane;
      const int c = __ffsll((long long)s + mm * S + 1) - 1;
      const unsigned bal = __ballot_sync(0xFFFFFFFFu, mm < Pm && c < 32 && ((any >> c) & 1u));
      if (!bal) {
        mi += 32;
        b0 = 0;
        continue;
      }
      const int f = __ffs(bal) - 1;
      if (f > 0) b0 = 0;
      mi += f;
      const int cc = __shfl_sync(0xFFFFFFFFu, c, f);
      unsigned hit = 0;
      for (; b0 < blocks; b0 += 32) {
        hit = __ballot_sync(0xFFFFFFFFu, b0 + lane < blocks && ((pos[b0 + lane] >> cc) & 1u));
        if (hit) break;
      }
      if (!hit) {
        ++mi;
        b0 = 0;
        continue;
      }
      b0 += __ffs(hit) - 1;
      const int k = cc + (b0 << 6);
      E += (double)g[k];
      flip(k);
      any = any_class();
      if (++b0 == blocks) {
        ++mi;
        b0 = 0;
      }
    }

    __syncthreads();  // the last toggle
    for (int q = threadIdx.x; q < blocks; q += blockDim.x)
      theta_out[(size_t)s * blocks + q] = bits[q];
    if (threadIdx.x == 0) energy_out[s] = (float)(spin ? E : E / 2.0);
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Descent: repeat (select the best single flip under the reference geometry,
// flip it if its value is > 0) until none improves or max_flips is reached.
//
// The chain of a flip - row load, update, selection over all n nodes - is
// serial, so the kernel is bound by its latency; a thread keeps the gains, bits
// and tie priorities of 4 NG nodes in registers and the selection goes through
// as few synchronisations as the size allows:
//  * one warp (n <= 128): two redux steps, no barrier;
//  * one CTA (to kDescentCta): each warp's best through shared memory, one barrier;
//  * a cluster (CL): behind one CTA barrier warp 0 sends the CTA's best to every
//    CTA with st.async, counted on that CTA's mbarrier; every warp waits for all
//    of them and reduces them itself. (Every warp sending its own best saved the
//    barrier, but the reduction of 64 arrivals took 10 to 20 % of a flip.) Two
//    slot arrays and mbarriers alternate: a CTA sends flip f + 2 only after every
//    CTA has sent f + 1, so all its warps have read f, and a slot is not
//    overwritten while it is read. A wait that runs out, which one warp or lane
//    may see alone, raises the CTA's flag of that exchange; the warp goes on with
//    what its slots hold (an older node of the graph, or none), every warp passes
//    one more CTA barrier, the next flip's or the one behind the loop, and reads
//    the flag behind it, so the CTA leaves together and the others follow by
//    their own waits.
// During the exchange each warp pulls its best's row into L2 when it is a new
// one: the next flips are mostly among the warps' bests. (Loading the last
// exchange's runners-up into registers as well gained nothing below 12000 nodes
// and cost 17 % at 4096, whose matrix stays in L2.) Times: see pqi_single_descent.
constexpr int DC_SLOTS = 16;  // CTAs of a cluster, or warps of the one CTA, at most

struct __align__(16) DescentBest {
  uint32_t hi;    // ordered float value (0: none selectable)
  uint32_t lo;    // tie priority, larger first; 0: never selected
  uint32_t node;  // node << 1 | its bit
  uint32_t pad;
};

// The best of the warp's lanes, in every lane (priorities are unique).
__device__ __forceinline__ DescentBest warp_best(const DescentBest& b) {
  DescentBest r;
  r.hi = __reduce_max_sync(0xFFFFFFFFu, b.hi);
  r.lo = __reduce_max_sync(0xFFFFFFFFu, b.hi == r.hi ? b.lo : 0u);
  const unsigned src = __ballot_sync(0xFFFFFFFFu, b.hi == r.hi && b.lo == r.lo);
  r.node = __shfl_sync(0xFFFFFFFFu, b.node, __ffs(src) - 1);
  r.pad = 0u;
  return r;
}

template <typename WT, int NG, bool CL>
__global__ void __launch_bounds__(512) descent_kernel(const WT* __restrict__ Wp, int ld, int n,
                                                      uint32_t* __restrict__ theta, double* __restrict__ g64,
                                                      int spin, SelGeom geo, int max_flips,
                                                      double* __restrict__ energy_sum, int* __restrict__ flips,
                                                      int* __restrict__ trace, int* __restrict__ status) {
  namespace cg = cooperative_groups;
  __shared__ DescentBest slots[2][DC_SLOTS];
  __shared__ __align__(8) uint64_t bar[2];
  __shared__ DescentBest wbest[DC_SLOTS];  // this CTA's warps
  __shared__ int wait_failed[2];           // by parity of the exchange
  __shared__ int any_failed;               // in rank 0: some CTA's wait ran out
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, T = blockDim.x, nwarps = T >> 5;
  int C = 1, rank = 0;
  if constexpr (CL) {
    C = (int)cg::this_cluster().num_blocks();
    rank = (int)cg::this_cluster().block_rank();
    if (threadIdx.x == 0) {
      tc::mbar_init(&bar[0], 1);
      tc::mbar_init(&bar[1], 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      wait_failed[0] = wait_failed[1] = any_failed = 0;
    }
    if (threadIdx.x < 2 * DC_SLOTS) slots[threadIdx.x & 1][threadIdx.x >> 1] = DescentBest{0u, 0u, 0u, 0u};
    cg::this_cluster().sync();
  }
  const int nslots = CL ? C : nwarps;
  const int v0 = 4 * (rank * NG * T + (int)threadIdx.x);  // group j starts at v0 + 4 T j
  typedef typename std::conditional<NG <= 8, uint32_t, uint64_t>::type Mask;  // a bit per node
  double g[4 * NG];
  uint32_t lo[4 * NG];
  Mask xm = 0;
#pragma unroll
  for (int j = 0; j < NG; ++j) {
    const int v = v0 + 4 * T * j;
    if (v < ((n + 31) & ~31)) xm |= (Mask)((theta[v >> 5] >> (v & 31)) & 15u) << (4 * j);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const bool in = v + i < n;
      g[4 * j + i] = in ? g64[v + i] : 0.0;
      lo[4 * j + i] = in ? (uint32_t)sel_key(0.0f, (uint64_t)(v + i), geo) : 0u;
    }
  }
  uint32_t seen = 0xFFFFFFFFu;
  double esum = 0.0;
  int cnt = 0, st = PQI_OK, failed = 0;
  // lane r's view of CTA r: this CTA's slot and the barrier of even exchanges
  uint32_t rslot = 0, rbar = 0;
  if (CL && lane < C) {
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rslot) : "r"(tc::smem_u32(&slots[0][rank])), "r"(lane));
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rbar) : "r"(tc::smem_u32(&bar[0])), "r"(lane));
  }
  for (int f = 0;; ++f) {
    // the thread's best, as floats (a -0 below a +0 does not matter here: only
    // values above 0 are taken); NaN compares false throughout
    float bv = -INFINITY;
    uint32_t bl = 0u, be = 0u;
#pragma unroll
    for (int e = 0; e < 4 * NG; ++e) {
      float v = (float)g[e];
      if (spin) v *= 2.0f;
      if (lo[e] != 0u && (v > bv || (v == bv && lo[e] > bl))) {
        bv = v;
        bl = lo[e];
        be = (uint32_t)(v0 + 4 * T * (e >> 2) + (e & 3)) << 1 | (uint32_t)((xm >> e) & 1u);
      }
    }
    DescentBest b{bl ? ord_f32(bv) : 0u, bl, be, 0u};
    b = warp_best(b);
    const DescentBest own = b;
    const int par = f & 1;
    if constexpr (CL) {
      if (threadIdx.x == 0) tc::mbar_expect_tx(&bar[par], (uint32_t)(C * sizeof(DescentBest)));
      if (lane == 0) wbest[warp] = b;
      __syncthreads();
      failed = wait_failed[par ^ 1];  // another warp's last wait ran out
      if (warp == 0) {
        b = warp_best(lane < nwarps ? wbest[lane] : DescentBest{0u, 0u, 0u, 0u});
        if (lane < C)
          asm volatile(
              "st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.u64 [%0], {%1, %2}, [%3];" ::"r"(
                  rslot + par * (uint32_t)sizeof(slots[0])),
              "l"((uint64_t)b.lo << 32 | b.hi), "l"((uint64_t)b.node), "r"(rbar + par * 8u)
              : "memory");
      }
      // a new best of this warp: its row into L2 (a hint)
      if (lane == 0 && own.hi > 0x80000000u && own.node >> 1 != seen) {
        seen = own.node >> 1;
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(Wp + (size_t)seen * ld),
                     "r"((uint32_t)(ld * (int)sizeof(WT)))
                     : "memory");
      }
      if (failed) break;
      if (!tc::mbar_wait_spin(&bar[par], (uint32_t)(f >> 1) & 1u)) wait_failed[par] = 1;
    } else if (nwarps > 1) {
      if (lane == 0) slots[par][warp] = b;
      __syncthreads();
    }
    if (CL || nwarps > 1) {
      b = warp_best(lane < nslots ? slots[par][lane] : DescentBest{0u, 0u, 0u, 0u});
    }
    const float val = b.lo ? unord_f32(b.hi) : -INFINITY;
    const bool none = !(val > 0.0f);
    if (none || cnt >= max_flips) {
      st = none ? PQI_OK : PQI_ETIMEOUT;
      if constexpr (CL) {
        __syncthreads();  // (the one that warps which go on pass in their next flip)
        failed = wait_failed[par];
      }
      break;
    }
    esum += (double)val;
    const int k = (int)(b.node >> 1);
    const uint32_t xk = b.node & 1u;
    if (rank == 0 && threadIdx.x == 0 && trace) trace[cnt] = k;
    ++cnt;
    const WT* __restrict__ row = Wp + (size_t)k * ld;
    WT w[4 * NG];
#pragma unroll
    for (int j = 0; j < NG; ++j) {
      const int v = v0 + 4 * T * j;
      if (v < n) {  // (rows are zero padded to a multiple of 128)
        if constexpr (sizeof(WT) == 4) {
          const float4 t = __ldg(reinterpret_cast<const float4*>(row + v));
          w[4 * j] = t.x; w[4 * j + 1] = t.y; w[4 * j + 2] = t.z; w[4 * j + 3] = t.w;
        } else {
          const char4 t = __ldg(reinterpret_cast<const char4*>(row + v));
          w[4 * j] = t.x; w[4 * j + 1] = t.y; w[4 * j + 2] = t.z; w[4 * j + 3] = t.w;
        }
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) w[4 * j + i] = (WT)0;
      }
    }
#pragma unroll
    for (int e = 0; e < 4 * NG; ++e) {
      const int v = v0 + 4 * T * (e >> 2) + (e & 3);
      const double w2 = 2.0 * (double)w[e];
      if (v == k) {
        g[e] = -g[e];
        xm ^= (Mask)1 << e;
      } else {
        g[e] += (uint32_t)((xm >> e) & 1u) == xk ? -w2 : w2;
      }
    }
  }
  // eight lanes assemble one word of 32 nodes
#pragma unroll
  for (int j = 0; j < NG; ++j) {
    const int v = v0 + 4 * T * j;
    uint32_t wd = ((uint32_t)(xm >> (4 * j)) & 15u) << (4 * (lane & 7));
    wd |= __shfl_xor_sync(0xFFFFFFFFu, wd, 1);
    wd |= __shfl_xor_sync(0xFFFFFFFFu, wd, 2);
    wd |= __shfl_xor_sync(0xFFFFFFFFu, wd, 4);
    if ((lane & 7) == 0 && v < n) theta[v >> 5] = wd;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (v + i < n) g64[v + i] = g[4 * j + i];
  }
  if constexpr (CL) {
    if (failed && threadIdx.x == 0) *cg::this_cluster().map_shared_rank(&any_failed, 0) = 1;
    cg::this_cluster().sync();  // (and no CTA leaves while another may still send to it)
    if (any_failed) st = PQI_ECUDA;
  }
  if (rank == 0 && threadIdx.x == 0) {
    *energy_sum = esum;
    *flips = cnt;
    *status = st;
  }
}

static size_t gray_smem_bytes(int n, size_t gain_bytes) {
  const int blocks = (n + 63) >> 6;
  return (((size_t)blocks * 12 + 15) & ~size_t(15)) + (size_t)n * gain_bytes;
}

static constexpr size_t kMaxGraySmem = 208 * 1024;

// Largest graph that descends in one CTA (512 threads of four nodes): at 2048
// nodes 0.90 us per flip against 1.01 with a cluster, at 4096 (two groups per
// thread) 1.32 against 0.96.
constexpr int kDescentCta = 2048;  // 512 * 4 at most

// CTAs of a descent's cluster: 16 where the device can place them.
static int descent_cluster() {
  static const int size = [] {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 16;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(512);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int fit = 0;
    const void* k = (const void*)descent_kernel<float, 16, true>;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&fit, k, &cfg) != cudaSuccess || fit < 1) {
      cudaGetLastError();
      return 8;
    }
    return 16;
  }();
  return size;
}

}  // namespace pqi

using namespace pqi;

extern "C" {

// 148 seeds, n^2 iterations in all, from a local optimum (microseconds, testing
// 32 positions per step -> now): complete float graphs of 1000 nodes 49 -> 39,
// 4096 464 -> 62, 8192 3282 -> 85, 24000 80750 -> 223; ER 2048 113 -> 56.
pqi_status pqi_gray(const pqi_weights* w, const uint64_t* theta64, const double* gains64,
                    int is_spin_glass, int iters_bound, int seeds, uint64_t* theta_out,
                    float* energy_out, void* workspace, size_t workspace_bytes, void* stream) {
  PQI_CHECK_ARG(w && theta64 && theta_out && energy_out && seeds > 0 && iters_bound >= 0);
  const int n = w->n;
  cudaStream_t s = as_stream(stream);
  Workspace ws(workspace, workspace_bytes);
  if (!gains64) {
    // gains of theta: unpack the 64-bit words as 32-bit words (same bit order)
    double* g = ws.take<double>(n);
    PQI_CHECK_ARG(g);
    pqi_status rc = launch_gains(w, reinterpret_cast<const uint32_t*>(theta64), 1, nullptr, g, s);
    if (rc) return rc;
    gains64 = g;
  }
  const bool i8 = w->kind == PQI_W_I8;
  const size_t gbytes = i8 ? sizeof(int) : sizeof(double);
  size_t smem = gray_smem_bytes(n, gbytes);
  int grid = seeds;
  void* gglob = nullptr;
  if (smem > kMaxGraySmem) {
    // gains in global memory, one n-vector per CTA
    smem = gray_smem_bytes(n, 0);
    PQI_CHECK_ARG(smem <= kMaxGraySmem);
    const size_t avail = (ws.size > ws.used + 256) ? (ws.size - ws.used - 256) : 0;
    const long long ctas = (long long)(avail / ((size_t)n * gbytes));
    PQI_CHECK_ARG(ctas >= 1);
    grid = (int)std::min<long long>(std::min<long long>(ctas, seeds), 148 * 4);
    gglob = ws.take<char>((size_t)grid * n * gbytes);
    PQI_CHECK_ARG(gglob);
  }
  if (i8) {
    PQI_TRY(cudaFuncSetAttribute(gray_kernel<int8_t>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
    gray_kernel<int8_t><<<grid, kGrayThreads, smem, s>>>(w->W_i8, w->ld, n, theta64, gains64,
                                                is_spin_glass, iters_bound, seeds, theta_out,
                                                energy_out, static_cast<int*>(gglob));
  } else {
    PQI_TRY(cudaFuncSetAttribute(gray_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
    gray_kernel<float><<<grid, kGrayThreads, smem, s>>>(w->W_f32z, w->ld, n, theta64, gains64,
                                               is_spin_glass, iters_bound, seeds, theta_out,
                                               energy_out, static_cast<double*>(gglob));
  }
  PQI_LAUNCHED("gray_kernel");
  return PQI_OK;
}

pqi_status pqi_single_descent(const pqi_weights* w, uint32_t* theta, double* gains64,
                              int is_spin_glass, int global_size, int local_size, int max_flips,
                              double* energy_sum, int* flips, int* trace, void* workspace,
                              size_t workspace_bytes, void* stream) {
  PQI_CHECK_ARG(w && theta && gains64 && energy_sum && flips && max_flips >= 0);
  const int n = w->n;
  SelGeom geo;
  PQI_CHECK_ARG(make_sel_geom(n, global_size, local_size, &geo));
  Workspace ws(workspace, workspace_bytes);
  int* status = ws.take<int>(1);
  PQI_CHECK_ARG(status);
  cudaStream_t s = as_stream(stream);
  // Threads of 4 NG nodes: one warp up to 128 nodes, one CTA up to kDescentCta,
  // else a cluster. Microseconds per flip, one CTA with the gains in shared
  // memory and the tie rule's divisions per node -> now: complete float graphs
  // of 300 nodes 2.8 -> 1.06, 1000 3.9 -> 0.85, 2048 4.5 -> 0.90, 4096 5.6 -> 0.96,
  // 8192 8.2 -> 1.12 (a whole descent 38.4 -> 5.3 ms), 16384 13.9 -> 1.20.
  const int groups = (n + 3) / 4;
  int C = 1, T = 32, NG = 1;
  auto shape = [&](int c, int tmax) {
    const int per = (groups + c - 1) / c;
    C = c;
    T = std::min(tmax, (per + 31) / 32 * 32);
    const int ng = (per + T - 1) / T;
    NG = ng <= 1 ? 1 : ng <= 2 ? 2 : ng <= 4 ? 4 : ng <= 8 ? 8 : ng <= 16 ? 16 : 0;
  };
  if (n <= 128) {
    shape(1, 32);
  } else if (n <= kDescentCta) {
    shape(1, 512);
  } else {
    const int c = descent_cluster();
    for (int tmax = 128; tmax <= 512; tmax *= 2) {  // fewest groups per thread first
      shape(c, tmax);
      if (NG == 1) break;
    }
  }
  PQI_CHECK_ARG(NG > 0);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.stream = s;
  auto launch = [&](auto kern, auto wp) -> pqi_status {
    if (C > 1) {
      PQI_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
      attr[0].val.clusterDim.x = C;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
    }
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(T);
    PQI_TRY(cudaLaunchKernelEx(&cfg, kern, wp, w->ld, n, theta, gains64, is_spin_glass, geo, max_flips, energy_sum,
                               flips, trace, status));
    return PQI_OK;
  };
  auto pick = [&](auto wp) -> pqi_status {
    typedef typename std::remove_const<typename std::remove_pointer<decltype(wp)>::type>::type WT;
    if (C == 1)
      return launch(descent_kernel<WT, 1, false>, wp);  // (512 threads of four nodes cover kDescentCta)
    return NG == 1   ? launch(descent_kernel<WT, 1, true>, wp)
           : NG == 2 ? launch(descent_kernel<WT, 2, true>, wp)
           : NG == 4 ? launch(descent_kernel<WT, 4, true>, wp)
           : NG == 8 ? launch(descent_kernel<WT, 8, true>, wp)
                     : launch(descent_kernel<WT, 16, true>, wp);  // (int8 past 262144 nodes)
  };
  const pqi_status rc = w->kind == PQI_W_I8 ? pick((const int8_t*)w->W_i8) : pick((const float*)w->W_f32z);
  if (rc != PQI_OK) return rc;
  PQI_LAUNCHED("descent_kernel");
  int hst = 0;
  PQI_TRY(cudaMemcpyAsync(&hst, status, sizeof(int), cudaMemcpyDeviceToHost, s));
  PQI_TRY(cudaStreamSynchronize(s));
  return (pqi_status)hst;
}

}  // extern "C"
