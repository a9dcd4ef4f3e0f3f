// libpqi: the TFIM-inspired candidate sampler of maxcut_tfim on the GPU
// (pyqrackising/maxcut_tfim.py:36-74, 139-145, 189-209 and
// maxcut_tfim_util.py:545-724).
//
//  * tfim_jz: per-node mean coupling J_eff and degree (init_J_and_z).
//  * tfim_cdf: the Hamming-weight distribution (maxcut_hamming_cdf with
//    probability_by_hamming_weight and _apply_time_envelope), float64: per
//    (step, node) pair the envelope's parameters in closed form, then per bin
//    the sum over pairs in a fixed order.
//  * tfim_sample: one warp per shot draws a Hamming weight from the CDF
//    (sample_mag) and picks nodes with multiplicative repulsion
//    (local_repulsion_choice, bit_pick), float64 weights so a weight that
//    underflows to zero counts as picked exactly as in the reference. The
//    selection mask is written as packed bits for the scoring kernel.
// Random numbers: a counter-based generator keyed by (seed, round, shot,
// draw), so a run is reproducible for a given seed (the reference's numba
// generator is unseeded and not reproducible, maxcut_tfim_util.py:692,715).
#include <algorithm>

#include "pqi_common.cuh"

namespace pqi {

constexpr double kEps = 1.1920928955078125e-07;  // float32 epsilon, the reference's `epsilon`
constexpr double kPi = 3.141592653589793;
constexpr double kLn2 = 0.6931471805599453;
constexpr double kLog2E = 1.4426950408889634;

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  // SplitMix64 finaliser (Steele, Lea, Flood 2014)
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// uniform double in [0, 1) from a counter
__device__ __forceinline__ double uniform(uint64_t seed, uint64_t round, uint64_t shot,
                                          uint64_t draw) {
  uint64_t h = mix64(seed ^ mix64(round * 0x632BE59BD9B4E019ull + shot));
  h = mix64(h ^ (draw * 0xD1B54A32D192ED03ull));
  return (double)(h >> 11) * (1.0 / 9007199254740992.0);
}

// ---------------------------------------------------------------------------
// init_J_and_z (maxcut_tfim.py:189-209): G_min over all of W (diagonal
// included); per row, entries with W - G_min > eps count as edges.

__global__ void tfim_min_kernel(const float* __restrict__ W, long long total, float* out_min) {
  __shared__ float red[32];
  float m = INFINITY;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x)
    m = fminf(m, W[e]);
  for (int o = 16; o > 0; o >>= 1) m = fminf(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 32) {
    m = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : INFINITY;
    for (int o = 16; o > 0; o >>= 1) m = fminf(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
    if (threadIdx.x == 0) {
      // order-preserving for floats of either sign: store as int via ordered key
      unsigned int k = __float_as_uint(m);
      k = (k & 0x80000000u) ? ~k : (k | 0x80000000u);
      atomicMin(reinterpret_cast<unsigned int*>(out_min), k);
    }
  }
}

__global__ void tfim_jz_kernel(const float* __restrict__ W, int n, const float* min_key,
                               double* __restrict__ J_eff, unsigned int* __restrict__ degrees) {
  unsigned int k = *reinterpret_cast<const unsigned int*>(min_key);
  k = (k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k;
  const float gmin = __uint_as_float(k);
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  for (int r = blockIdx.x * warps + (threadIdx.x >> 5); r < n; r += gridDim.x * warps) {
    const float* row = W + (size_t)r * n;
    unsigned int deg = 0;
    double J = 0.0;
    for (int m = lane; m < n; m += 32) {
      const float val = row[m] - gmin;  // float32, as the reference
      if ((double)val <= kEps) continue;
      ++deg;
      J += (double)val;
    }
    for (int o = 16; o > 0; o >>= 1) {
      deg += __shfl_xor_sync(0xFFFFFFFFu, deg, o);
      J += __shfl_xor_sync(0xFFFFFFFFu, J, o);
    }
    if (lane == 0) {
      J_eff[r] = deg > 0 ? -J / (double)deg : 0.0;
      degrees[r] = deg;
    }
  }
}

// The sparse path's J_eff and degrees (maxcut_tfim_sparse.py:204-224): the
// same rule, but the reference runs it as plain numpy scalar arithmetic, so
// the row sum is float32, accumulated in node order, and J = -(sum / degree)
// is a float32 division. One thread per row reproduces that order exactly.
__global__ void tfim_jz_f32_kernel(const float* __restrict__ W, int n, const float* min_key,
                                   double* __restrict__ J_eff, unsigned int* __restrict__ degrees) {
  unsigned int k = *reinterpret_cast<const unsigned int*>(min_key);
  k = (k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k;
  const float gmin = __uint_as_float(k);
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    const float* row = W + (size_t)r * n;
    unsigned int deg = 0;
    float J = 0.0f;
    for (int m = 0; m < n; ++m) {
      const float val = __fsub_rn(row[m], gmin);
      if ((double)val <= kEps) continue;
      ++deg;
      J = __fadd_rn(J, val);
    }
    J_eff[r] = deg > 0 ? (double)(-__fdiv_rn(J, (float)deg)) : 0.0;
    degrees[r] = deg;
  }
}

// ---------------------------------------------------------------------------
// maxcut_hamming_cdf (maxcut_tfim_util.py:654-687)

struct CdfParams {
  int n;           // nodes; bins are 0..n
  int n_steps;     // 1 << quality
  double delta_t;  // tot_t / n_steps
  double tot_t;
  double h_mult;   // |anneal_h|
  double omega;
};

// p of probability_by_hamming_weight (util:627-631) for node q at time t
__device__ __forceinline__ double pbhw_p(double J, double h, double z, double theta, double t,
                                         double omega) {
  const double zJ = z * J;
  const double theta_c =
      fabs(zJ) < kEps ? ((J > 0 ? kPi : -kPi) / 2) : asin(fmax(-1.0, fmin(1.0, h / zJ)));
  return exp2(fabs(J / h) - 1.0) *
             (1.0 + sin(theta - theta_c) * cos(omega * J * t + theta) / (1.0 + sqrt(t))) -
         0.5;
}

// The envelope of a (step, node) pair at time tt (util:596-651): with b = -p /
// (n + 1) and a = log2(e) / t_eff, bin k holds 2^e(k) / Z, e(k) = b (k + 1) -
// a |k - n/2| and Z = sum_k 2^e(k) (the normaliser of the bias alone cancels).
// e is linear on each side of n/2, so Z is two geometric sums: O(1) per pair
// instead of a pass over the n + 1 bins. All exponents are taken relative to
// the bin of the largest one (an end or next to n/2), so nothing overflows;
// where that largest term underflows in the reference's arithmetic (or b is
// not finite) the distribution is the delta at half filling (util:612-618):
// iz < 0; skipped nodes have iz = 0.
struct CdfEnv {
  double b;   // log2 of the bias ratio of neighbouring bins
  double a;   // log2(e) / t_eff
  double k0;  // the bin of the largest exponent
  double iz;  // 1 / Z relative to that bin
  double r;   // ratio of neighbouring bins going away from n/2 (on one side)
};

// sum_{i < m} 2^(-s i), s >= 0
__device__ __forceinline__ double geo_sum(double s, int m) {
  const double x = -s * kLn2;
  return x == 0.0 ? (double)m : expm1((double)m * x) / expm1(x);
}

// e(k) - e(k0) for the bin k0 of the largest exponent: the differences are
// formed before the products, so bins near k0 keep full precision.
__device__ __forceinline__ double env_exp(double b, double a, double half, int k, int k0) {
  return b * (double)(k - k0) - a * (fabs((double)k - half) - fabs((double)k0 - half));
}

// The bin of the largest exponent: e is concave, so an end or next to n/2.
__device__ __forceinline__ int env_peak(double b, double a, int n) {
  const int kl = n / 2;  // floor(n/2); kl + 1 is as far from n/2 for odd n
  if (b > a) return n;
  if (b < -a) return 0;
  return (n & 1) && b > 0.0 ? kl + 1 : kl;
}

// The envelope of node q at step and time t (which = 0) or t - dt (1), for the
// bins below (left) or above n/2. J_eff = -(mean positive excess) <= 0, so the
// reversed, unnormalised J > 0 branch of probability_by_hamming_weight never
// applies.
__device__ __forceinline__ CdfEnv cdf_env(const CdfParams& P, double J, double z, int step, int which,
                                          bool left) {
  CdfEnv o{0.0, 0.0, 0.0, 0.0, 0.0};
  if (fabs(J) < kEps) return o;
  const int n = P.n;
  const double half = n / 2.0;
  const double zJ0 = z * J;
  const double theta =
      fabs(zJ0) < kEps ? ((J > 0 ? kPi : -kPi) / 2) : asin(fmax(-1.0, fmin(1.0, P.h_mult / zJ0)));
  const double t = step * P.delta_t, tt = which == 0 ? t : (step - 1) * P.delta_t;
  const double h_t = P.h_mult * (P.tot_t - t);
  o.b = -pbhw_p(J, h_t, z, theta, tt, P.omega) / (n + 1);
  o.a = kLog2E / (tt > 1e-9 ? tt : 1e-9);
  const int k0 = env_peak(o.b, o.a, n);
  o.k0 = (double)k0;
  // the reference's largest bin underflows to zero below 2^-1075
  const double top = o.b * (double)(k0 + 1) - o.a * fabs((double)k0 - half);
  if (!(top >= -1075.0) || isinf(o.b)) {
    o.iz = -1.0;
    return o;
  }
  const int kl = n / 2, ml = kl + 1, mr = n - kl;
  const double sl = o.b + o.a, sr = o.a - o.b;  // decrease per bin going down / up
  // each side summed from its larger end
  const double el = env_exp(o.b, o.a, half, sl >= 0.0 ? kl : 0, k0);
  const double er = env_exp(o.b, o.a, half, sr >= 0.0 ? kl + 1 : n, k0);
  o.iz = 1.0 / (exp2(el) * geo_sum(fabs(sl), ml) + exp2(er) * geo_sum(fabs(sr), mr));
  o.r = exp2(left ? -sl : -sr);
  return o;
}

// hamming_prob[k] += envelope(t)[k] - envelope(t - dt)[k] over the pairs
// (util:675-676). Compute bound (float64). A thread owns CDF_BINS consecutive
// bins of one side of n/2, counted away from it, so an envelope costs it one
// exp2 and then a multiply per bin (the ratio of neighbours); CDF_BINS
// multiplies add at most that many roundings to a bin. A block takes a
// contiguous slice of the pairs in tiles of CDF_THREADS envelopes: each thread
// works out one envelope into shared memory, then all threads walk the tile
// (the envelopes are recomputed per block of bins: cheaper than a pass through
// memory, and no buffer that grows with the pairs). The slices' partial sums
// are added in order by the next kernel. Times: see pqi_tfim_cdf.
constexpr int CDF_BINS = 8;
constexpr int CDF_THREADS = 128;
constexpr int CDF_BLOCK_BINS = CDF_BINS * CDF_THREADS;
// ratios steeper than 2^-64 per bin (a start value could underflow while a
// later bin does not): every bin from its own exp2
constexpr double kSteep = 64.0;

__global__ void __launch_bounds__(CDF_THREADS) tfim_cdf_accum_kernel(CdfParams P, const double* __restrict__ J_eff,
                                                                     const unsigned int* __restrict__ degrees,
                                                                     long long pairs_per_slice,
                                                                     double* __restrict__ partial) {
  __shared__ CdfEnv tile[CDF_THREADS];
  const int n = P.n, kl = n / 2;
  const double half = n / 2.0;
  const int left_blocks = (kl + CDF_BLOCK_BINS) / CDF_BLOCK_BINS;  // covers kl + 1 bins
  const bool left = (int)blockIdx.x < left_blocks;
  const int i0 = (left ? blockIdx.x : blockIdx.x - left_blocks) * CDF_BLOCK_BINS + threadIdx.x * CDF_BINS;
  const int bins = left ? kl + 1 : n - kl;
  const int cnt = min(CDF_BINS, bins - i0);  // may be <= 0: the thread only fills tiles
  const int kfirst = left ? kl - i0 : kl + 1 + i0, dir = left ? -1 : 1;
  const double dfirst = fabs((double)kfirst - half);
  const long long pairs = (long long)(P.n_steps - 1) * n;
  const long long p0 = blockIdx.y * pairs_per_slice;
  const long long p1 = p0 + pairs_per_slice < pairs ? p0 + pairs_per_slice : pairs;
  double acc[CDF_BINS];
#pragma unroll
  for (int i = 0; i < CDF_BINS; ++i) acc[i] = 0.0;
  for (long long pt = p0; pt < p1; pt += CDF_THREADS / 2) {
    __syncthreads();  // the previous tile's reads are done
    {
      const long long pr = pt + (threadIdx.x >> 1);
      CdfEnv e{0.0, 0.0, 0.0, 0.0, 0.0};
      if (pr < p1) {
        const int step = 1 + (int)(pr / n), q = (int)(pr % n);
        e = cdf_env(P, J_eff[q], (double)degrees[q], step, threadIdx.x & 1, left);
      }
      tile[threadIdx.x] = e;
    }
    __syncthreads();
    if (cnt <= 0) continue;
    const int m = 2 * (int)(p1 - pt < CDF_THREADS / 2 ? p1 - pt : CDF_THREADS / 2);
    for (int it = 0; it < m; ++it) {
      const CdfEnv& e = tile[it];
      double iz = e.iz;
      if (iz == 0.0) continue;  // skipped node
      if (iz < 0.0) {           // delta at half filling
        if (left && i0 == 0) acc[0] += (it & 1) ? -1.0 : 1.0;
        continue;
      }
      if (it & 1) iz = -iz;  // envelope(t - dt) is subtracted
      const double x0 = e.b * ((double)kfirst - e.k0) - e.a * (dfirst - fabs(e.k0 - half));
      const double r = e.r;
      if (fabs(left ? e.b + e.a : e.a - e.b) < kSteep) {
        if (x0 < -1100.0 && !(r > 1.0)) continue;  // this and every later bin underflow
        double v = exp2(x0) * iz;
#pragma unroll
        for (int i = 0; i < CDF_BINS; ++i) {
          acc[i] += v;
          v *= r;
        }
      } else {
#pragma unroll 1
        for (int i = 0; i < CDF_BINS; ++i) {
          const double v = exp2(env_exp(e.b, e.a, half, kfirst + dir * i, (int)e.k0)) * iz;
#pragma unroll
          for (int j = 0; j < CDF_BINS; ++j)
            if (j == i && i < cnt) acc[j] += v;
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < CDF_BINS; ++i)
    if (i < cnt) partial[(size_t)blockIdx.y * (n + 1) + kfirst + dir * i] = acc[i];
}

// hprob[k] = start[k] + the slices' partial sums, eight threads per bin.
__global__ void __launch_bounds__(256) tfim_cdf_reduce_kernel(int n, int slices, const double* __restrict__ start,
                                                              const double* __restrict__ partial,
                                                              double* __restrict__ hprob) {
  __shared__ double red[8][33];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const int k = blockIdx.x * 32 + x;
  double s = 0.0;
  if (k <= n)
    for (int j = y; j < slices; j += 8) s += partial[(size_t)j * (n + 1) + k];
  red[y][x] = s;
  __syncthreads();
  if (y == 0 && k <= n) {
    for (int j = 1; j < 8; ++j) s += red[j][x];
    hprob[k] = start[k] + s;
  }
}

// normalise and accumulate the CDF over bins 1..n-1 (util:678-687); one block:
// each thread sums a contiguous run of bins, the runs' totals are scanned.
__global__ void __launch_bounds__(1024) tfim_cdf_finish_kernel(int n, const double* __restrict__ hprob,
                                                               double* __restrict__ cum) {
  __shared__ double wsum[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int m = n - 1;  // bins 1 .. n-1
  const int per = (m + 1023) / 1024;
  const int i0 = min(m, (int)threadIdx.x * per), i1 = min(m, i0 + per);
  double tot = 0.0, run = 0.0;
  // pass 0: the sum of all bins (the normaliser); pass 1: the scan
  for (int pass = 0; pass < 2; ++pass) {
    double s = 0.0;
    for (int i = i0; i < i1; ++i) s += pass == 0 ? hprob[i + 1] : hprob[i + 1] / tot;
    double x = s;
    for (int o = 1; o < 32; o <<= 1) {
      const double y = __shfl_up_sync(0xFFFFFFFFu, x, o);
      if (lane >= o) x += y;
    }
    __syncthreads();
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    double w = wsum[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const double y = __shfl_up_sync(0xFFFFFFFFu, w, o);
      if (lane >= o) w += y;
    }
    tot = pass == 0 ? __shfl_sync(0xFFFFFFFFu, w, 31) : tot;
    const double before = __shfl_sync(0xFFFFFFFFu, w, (warp + 31) & 31);
    run = (warp > 0 ? before : 0.0) + (x - s);
  }
  for (int i = i0; i < i1; ++i) {
    run += hprob[i + 1] / tot;
    cum[i] = i == m - 1 ? 1.0 : run;
  }
}

// ---------------------------------------------------------------------------
// Sampler: one warp per shot; lane l owns nodes [l*C, (l+1)*C), C = ceil(n/32).

// sample_mag (util:691-707), step for step: bisect for an m with cum[m] >= p
// and (m == 0 or cum[m-1] < p). The reference's cumulative array need not be
// monotone (it accumulates differences of distributions), so this is not a
// plain lower bound; the same probes give the same m. The loop is capped at 64
// probes (the reference loops until the condition holds).
__device__ __forceinline__ int sample_mag(const double* cum, int len, double p) {
  int left = 0, right = len - 1, m = 0;
  for (int it = 0; it < 64; ++it) {
    m = (left + right) >> 1;
    if (cum[m] >= p && (m == 0 || cum[m - 1] < p)) break;
    if (cum[m] < p) {
      left = m + 1;
    } else {
      right = m - 1;
    }
  }
  return m;
}

constexpr int kWtsPitch = 33;  // doubles per row of a warp's weight table (32 lanes + 1)
constexpr int kRowBatch = 16;  // row steps of 32 weights in flight per repulsion update

// base^(-w) for a weight other than +-1, out of line: the unrolled update loop
// stays small enough for the instruction cache
__device__ __noinline__ double repulsion_factor(double lnb, float wv) {
  return exp(-lnb * (double)wv);
}

// adj_ptr / adj_col / adj_val (nullable): the nonzero entries of each row of W
// in column order; when given, a repulsion update walks the picked node's
// list instead of scanning its dense row (the same multiplications).
__global__ void tfim_sample_kernel(const float* __restrict__ W, int n,
                                   const double* __restrict__ cum, int ncum, double base,
                                   int repel, uint64_t seed, uint64_t round, int shots,
                                   uint32_t* __restrict__ theta_out, double* __restrict__ wglob,
                                   int use_smem, const long long* __restrict__ adj_ptr,
                                   const int* __restrict__ adj_col,
                                   const float* __restrict__ adj_val) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const int wpb = blockDim.x >> 5;
  const int C = (n + 31) >> 5;
  const int n32 = C;  // words per packed row == nodes per lane chunk, both ceil(n/32)
  double* wts = use_smem ? reinterpret_cast<double*>(smem) + (size_t)wib * (C * kWtsPitch)
                         : wglob + (size_t)(blockIdx.x * wpb + wib) * (C * kWtsPitch);
  const double lnb = log(base);
  const double rep1 = exp(-lnb);  // repulsion factors of the weights +1 and -1
  const double repm1 = exp(lnb);
  for (int s = blockIdx.x * wpb + wib; s < shots; s += gridDim.x * wpb) {
    const int m = sample_mag(cum, ncum, uniform(seed, round, (uint64_t)s, 0));
    const int node0 = s % n;
    uint32_t* out = theta_out + (size_t)s * n32;
    if (m == 1) {
      for (int w = lane; w < n32; w += 32) out[w] = (w == (node0 >> 5)) ? (1u << (node0 & 31)) : 0u;
      continue;
    }
    // lane l owns nodes v0 .. v0 + C - 1 (the bisection's order); node v0 + i
    // is stored at wts[i * 33 + l]: the owners' sweeps (fixed i, 32 lanes) and
    // the node-order sweeps (32 consecutive nodes) both spread over the banks
    const int v0 = lane * C;
    for (int i = 0; i < C; ++i) wts[i * kWtsPitch + lane] = (v0 + i < n) ? 1.0 : 0.0;
    __syncwarp();
    // picks after the first node: m - 1 for m >= 2, one for m == 0 (the loop of
    // local_repulsion_choice runs max(0, m - 2) times, then one last pick)
    const int picks = (m == 0) ? 1 : m - 1;
    int node = node0;
    for (int j = 0; j <= picks; ++j) {
      if (j > 0) {
        // bit_pick (util:711-724): p = sum(weights) * u, first i with p < running sum.
        // The lane's sum runs as four interleaved partial sums (independent
        // adds instead of one chain of C).
        double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
        int i = 0;
        for (; i + 3 < C; i += 4) {
          a0 += wts[i * kWtsPitch + lane];
          a1 += wts[(i + 1) * kWtsPitch + lane];
          a2 += wts[(i + 2) * kWtsPitch + lane];
          a3 += wts[(i + 3) * kWtsPitch + lane];
        }
        for (; i < C; ++i) a0 += wts[i * kWtsPitch + lane];
        const double loc = (a0 + a1) + (a2 + a3);
        double incl = loc;
        for (int o = 1; o < 32; o <<= 1) {
          const double y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
          if (lane >= o) incl += y;
        }
        const double total = __shfl_sync(0xFFFFFFFFu, incl, 31);
        const double p = total * uniform(seed, round, (uint64_t)s, (uint64_t)j);
        const unsigned hit = __ballot_sync(0xFFFFFFFFu, p < incl);
        int picked = 0;
        if (hit) {
          // lane l's chunk holds the pick: the whole warp scans its C weights,
          // 32 at a time (inclusive warp scan on top of the running sum)
          const int l = __ffs(hit) - 1;
          double run = __shfl_sync(0xFFFFFFFFu, incl - loc, l);
          picked = l * C;  // no prefix above p (rounding): the chunk's first node
          for (int i0 = 0; i0 < C; i0 += 32) {
            const int ii = i0 + lane;
            double w = (ii < C) ? wts[ii * kWtsPitch + l] : 0.0;
            for (int o = 1; o < 32; o <<= 1) {
              const double y = __shfl_up_sync(0xFFFFFFFFu, w, o);
              if (lane >= o) w += y;
            }
            const unsigned h2 = __ballot_sync(0xFFFFFFFFu, ii < C && p < run + w);
            if (h2) {
              picked = l * C + i0 + __ffs(h2) - 1;
              break;
            }
            run += __shfl_sync(0xFFFFFFFFu, w, 31);
          }
          // the lanes' prefixes are summed in different orders, so one without
          // nodes may be above p by a rounding: as if none were
          if (picked >= n) picked = 0;
        }
        node = picked;
      }
      // update_repulsion_choice (maxcut_tfim.py:37-45) for all but the last pick
      __syncwarp();
      if (lane == (node / C)) wts[(node - lane * C) * kWtsPitch + lane] = 0.0;
      __syncwarp();
      if (j < picks && repel && adj_ptr) {
        // the picked node's nonzero weights, 32 list entries per step
        const long long e1 = adj_ptr[node + 1];
        for (long long e = adj_ptr[node] + lane; e < e1; e += 32) {
          const int v = adj_col[e];
          const float wv = adj_val[e];
          const int q = v / C;
          wts[(v - q * C) * kWtsPitch + q] *= (wv == 1.0f)    ? rep1
                                              : (wv == -1.0f) ? repm1
                                                              : repulsion_factor(lnb, wv);
        }
      } else if (j < picks && repel) {
        // the row in node order, 32 consecutive weights per step (coalesced),
        // kRowBatch steps loaded before any is applied (the weight table may
        // be global memory, so loads would otherwise wait behind the stores);
        // each lane scales the weight of its node v wherever v's owner keeps it
        const float* row = W + (size_t)node * n;
        int q = lane / C, r = lane - q * C;  // v = lane + 32 w = q C + r
        const int dq = 32 / C, dr = 32 - dq * C;
        for (int vb = lane; vb < n; vb += 32 * kRowBatch) {
          float wv[kRowBatch];
#pragma unroll
          for (int u = 0; u < kRowBatch; ++u) wv[u] = (vb + 32 * u < n) ? __ldg(row + vb + 32 * u) : 0.0f;
#pragma unroll
          for (int u = 0; u < kRowBatch; ++u) {
            if (wv[u] != 0.0f)
              wts[r * kWtsPitch + q] *= (wv[u] == 1.0f)    ? rep1
                                        : (wv[u] == -1.0f) ? repm1
                                                           : repulsion_factor(lnb, wv[u]);
            q += dq;
            r += dr;
            if (r >= C) {
              r -= C;
              ++q;
            }
          }
        }
      }
      __syncwarp();
    }
    // selection mask: weights == 0 (picked, or underflowed to zero)
    for (int w = 0; w < n32; ++w) {
      const int v = w * 32 + lane;
      const bool sel = v < n && wts[(v % C) * kWtsPitch + v / C] == 0.0;
      const unsigned bits = __ballot_sync(0xFFFFFFFFu, sel);
      if (lane == 0) out[w] = bits;
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// Register form of the sampler, n <= 2048: one warp per shot, lane l owns the
// nodes [l C, (l + 1) C) (C = ceil(n / 32) rounded up to a group) and keeps
// their float64 weights in registers, in groups of SR_GS whose sums it also
// keeps. A pick is then: the lanes' totals scanned over the warp, the owner of
// the hit found by ballot, its node by halving (each decision is the owner's,
// broadcast by a vote, so the branches are uniform and the registers' indices
// known at compile time), and one pass over the groups that the picked row
// touches - multiply and re-sum, never a running difference. The form above
// moves every weight through shared memory three times per pick (its bound);
// here a weight costs one predicated float64 multiply and one add, and the
// bound is instruction issue. Picks multiply each weight by the same factors
// in the same order as above, so the weights are the same numbers; only the
// order of the sums differs.
//
// The rows come as tables built from W at the start of the call, in the
// workspace (nothing is kept between calls): bit planes for weights in {0, +1,
// -1}, else the float64 factor of every entry. Control words tell which form
// the weights call for, so nothing is read back to the host: the kernels of the
// other forms return at once. Times: see tfim_sample_impl.
constexpr int SR_GS = 8;           // nodes per group
constexpr int SR_MAX_N = 32 * 64;  // C <= 64

// Sparse form (below): row slots
constexpr int SP_DEG = 15;
constexpr int SP_CODE_DEG = 7;

struct __align__(16) SparseEntry {
  double factor;
  int col;    // the row's own node for an empty slot
  int minus;  // weight -1
};

// Control words: some weight is -1; some weight is not in {0, +1, -1}; nonzero
// weights; the largest number of them in a row; some row of few has an entry
// whose mirror image is zero, so a column may be fuller than every row.
struct SampleCtl {
  unsigned minus, other, count, degree, lopsided;
};

// Tables of W's rows, a warp per row through shared memory:
//  * planes +1, -1, nonzero (n * 32 * NW words each): row r, lane l: NW =
//    ceil(C / 32) words of the lane's C nodes, lowest first;
//  * table (nullable): factors (1 where the weight is 0), row r as C / 2 runs
//    of 32 lanes x 2 nodes: lane l's nodes l C + 2 q and + 1 at (32 q + l) * 2,
//    so a warp of the sampler reads a run as one contiguous 512 bytes;
//  * slots (nullable): the first SP_DEG nonzero weights in column order.
// One block sets the control words itself; more add to zeroed ones.
__global__ void __launch_bounds__(1024) tfim_rows_kernel(const float* __restrict__ W, int n, int C, double base,
                                 uint32_t* __restrict__ planes, double* __restrict__ table,
                                 SparseEntry* __restrict__ slots, SampleCtl* __restrict__ ctl) {
  extern __shared__ float rows_smem[];
  __shared__ SampleCtl sc;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  const int NW = (C + 31) / 32, plane = n * 32 * NW;
  float* buf = rows_smem + (size_t)wib * 32 * (C + 1);  // node v at v + v / C: lanes on distinct banks
  const double lnb = log(base);
  const double rep1 = exp(-lnb), repm1 = exp(lnb);
  auto factor = [&](float w) {
    return w == 0.0f ? 1.0 : w == 1.0f ? rep1 : w == -1.0f ? repm1 : repulsion_factor(lnb, w);
  };
  if (threadIdx.x == 0) sc = SampleCtl{0u, 0u, 0u, 0u, 0u};
  __syncthreads();
  unsigned minus_any = 0, other = 0, count = 0, degree = 0, lopsided = 0;
  for (int r = blockIdx.x * wpb + wib; r < n; r += gridDim.x * wpb) {
    const float* row = W + (size_t)r * n;
    int at = 0;
    for (int v = lane; v < 32 * C; v += 32) {
      const float w = v < n ? __ldg(row + v) : 0.0f;
      buf[v + v / C] = w;
      const unsigned nz = __ballot_sync(0xFFFFFFFFu, w != 0.0f);
      if (slots && w != 0.0f) {
        const int e = at + __popc(nz & ((1u << lane) - 1u));
        if (e < SP_DEG) slots[(size_t)r * SP_DEG + e] = SparseEntry{factor(w), v, w == -1.0f};
        // (only as many as a row may have for the codes: a dozen loads per row)
        if (e < SP_CODE_DEG && __ldg(W + (size_t)v * n + r) == 0.0f) lopsided = 1;
      }
      at += __popc(nz);
    }
    if (slots && lane >= at && lane < SP_DEG) slots[(size_t)r * SP_DEG + lane] = SparseEntry{1.0, r, 0};
    degree = max(degree, (unsigned)at);
    count += lane == 0 ? at : 0;
    __syncwarp();
    for (int q = 0; q < NW; ++q) {
      uint32_t plus = 0, minus = 0, nz = 0;
      for (int i = 0; i < min(32, C - 32 * q); ++i) {
        const float w = buf[lane * (C + 1) + 32 * q + i];
        if (w == 1.0f) plus |= 1u << i;
        if (w == -1.0f) minus |= 1u << i;
        if (w != 0.0f) nz |= 1u << i;
      }
      const int e = (r * 32 + lane) * NW + q;
      planes[e] = plus;
      planes[plane + e] = minus;
      planes[2 * plane + e] = nz;
      minus_any |= minus;
      other |= nz & ~(plus | minus);
    }
    if (table)
      for (int x = lane; x < 32 * C; x += 32) {
        const int v = ((x >> 1) & 31) * C + 2 * (x >> 6) + (x & 1);
        table[(size_t)r * (32 * C) + x] = factor(buf[v + v / C]);
      }
    __syncwarp();
  }
  if (minus_any) atomicOr(&sc.minus, 1u);
  if (other) atomicOr(&sc.other, 1u);
  if (count) atomicAdd(&sc.count, count);
  if (lane == 0) atomicMax(&sc.degree, degree);
  if (lopsided) atomicOr(&sc.lopsided, 1u);
  __syncthreads();
  if (threadIdx.x == 0) {
    if (gridDim.x == 1) {
      *ctl = sc;
    } else {
      if (sc.minus) atomicOr(&ctl->minus, 1u);
      if (sc.other) atomicOr(&ctl->other, 1u);
      atomicAdd(&ctl->count, sc.count);
      atomicMax(&ctl->degree, sc.degree);
      if (sc.lopsided) atomicOr(&ctl->lopsided, 1u);
    }
  }
}

// Which form the weights call for. codes / lists: the sparse forms are there
// (chosen by n in tfim_sample_impl). A node's factors come by its column, so its
// code holds them all only where the columns are no fuller than the rows: the
// pattern of the weights must be its own mirror image (the caller's W need not
// be symmetric).
enum SampleForm { SF_BITS, SF_TABLE, SF_LISTS, SF_CODES };
__device__ __forceinline__ SampleForm sample_form(const SampleCtl& c, bool codes, bool lists) {
  if (codes && !c.other && !c.lopsided && c.degree <= SP_CODE_DEG) return SF_CODES;
  if (lists && c.degree <= SP_DEG) return SF_LISTS;
  return c.other ? SF_TABLE : SF_BITS;
}

// w *= f where bit != 0. The jump makes it one predicated multiply; written as
// a conditional it became a multiply and two selects (ER n = 1024, 32768
// shots: 10.0 ms against 7.6 ms).
__device__ __forceinline__ void mul_if(double& w, uint32_t bit, double f) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %1, 0;\n\t@p bra SKIP;\n\tmul.rn.f64 %0, %0, %2;\n\tSKIP:\n\t}"
      : "+d"(w)
      : "r"(bit), "d"(f));
}

// Inclusive scan over the warp: a lane's sum with the lanes below it (the
// shuffle's own predicate says whether there is one).
__device__ __forceinline__ double warp_scan(double x) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1)
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b32 lo, hi;\n\t.reg .f64 y;\n\t"
        "mov.b64 {lo, hi}, %0;\n\t"
        "shfl.sync.up.b32 lo, lo, %1, 0, 0xFFFFFFFF;\n\t"
        "shfl.sync.up.b32 hi|p, hi, %1, 0, 0xFFFFFFFF;\n\t"
        "mov.b64 y, {lo, hi};\n\t"
        "@!p bra SKIP;\n\tadd.rn.f64 %0, %0, y;\n\tSKIP:\n\t}"
        : "+d"(x)
        : "r"(o));
  return x;
}

// w[LO] + ... + w[LO + N - 1], pairwise
template <int LO, int N, int C>
__device__ __forceinline__ double tree_sum(const double (&w)[C]) {
  if constexpr (N == 1) {
    return w[LO];
  } else {
    return tree_sum<LO, (N + 1) / 2, C>(w) + tree_sum<LO + (N + 1) / 2, N / 2, C>(w);
  }
}

// The owner's node holding q among w[LO .. LO + N): its index, and its weight
// becomes zero. Groups are passed over by their sums, then the nodes of one.
template <int LO, int N, int C>
__device__ __forceinline__ int pick_node(double (&w)[C], const double (&sum)[C / SR_GS], double q, int owner,
                                         int lane) {
  if constexpr (N == 1) {
    if (lane == owner) w[LO] = 0.0;
    return LO;
  } else {
    constexpr int H = N > SR_GS ? (N / SR_GS + 1) / 2 * SR_GS : N / 2;
    double m;
    if constexpr (N > SR_GS) {
      m = tree_sum<LO / SR_GS, H / SR_GS, C / SR_GS>(sum);
    } else {
      m = tree_sum<LO, H, C>(w);
    }
    const unsigned below = __ballot_sync(0xFFFFFFFFu, q < m);
    if ((below >> owner) & 1u) return pick_node<LO, H, C>(w, sum, q, owner, lane);
    return pick_node<LO + H, N - H, C>(w, sum, q - m, owner, lane);
  }
}

// Resident blocks of 64 threads per SM, by measurement (ER and complete graphs
// of 32 C nodes): the latency of a pick wants warps, the weights want 2 C
// registers; a few spilled words cost less than a block, and the factor loads
// of TABLE need more registers in flight.
constexpr int sr_blocks(int C, bool table) {
  return C >= 56 ? 6 : C >= 48 ? (table ? 6 : 7) : C >= 40 ? 8 : C >= 32 ? 10 : C >= 24 ? (table ? 10 : 14) : (table && C >= 16 ? 14 : 16);
}

template <int C, bool TABLE>
__global__ void __launch_bounds__(64, sr_blocks(C, TABLE))
    tfim_sample_reg_kernel(int n, const double* __restrict__ cum, int ncum, double base, int repel, uint64_t seed,
                           uint64_t round, int shots, uint32_t* __restrict__ theta_out,
                           const uint32_t* __restrict__ planes, const double* __restrict__ table,
                           const SampleCtl* __restrict__ ctl, bool codes, bool lists) {
  constexpr int NG = C / SR_GS, NW = (C + 31) / 32;
  const SampleCtl ct = *ctl;
  if (sample_form(ct, codes, lists) != (TABLE ? SF_TABLE : SF_BITS)) return;
  const bool has_minus = ct.minus != 0;
  // factors of sparse rows are loaded one by one where the weight is not zero
  const bool sparse = (long long)ct.count * 4 < (long long)n * n;
  const int lane = threadIdx.x & 31;
  const int n32 = (n + 31) >> 5;
  const double lnb = log(base);
  const double rep1 = exp(-lnb), repm1 = exp(lnb);
  const int warps = (gridDim.x * blockDim.x) >> 5;
  const int plane = n * 32 * NW;
  for (int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < shots; s += warps) {
    const uint64_t key = mix64(seed ^ mix64(round * 0x632BE59BD9B4E019ull + (uint64_t)s));
    // uniform(seed, round, s, draw) with the shot's part worked out once
    auto draw = [&](int d) {
      const uint64_t h = mix64(key ^ ((uint64_t)d * 0xD1B54A32D192ED03ull));
      return (double)(h >> 11) * (1.0 / 9007199254740992.0);
    };
    const int m = sample_mag(cum, ncum, draw(0));
    int node = s % n;
    uint32_t* out = theta_out + (size_t)s * n32;
    if (m == 1) {
      for (int w = lane; w < n32; w += 32) out[w] = (w == (node >> 5)) ? (1u << (node & 31)) : 0u;
      continue;
    }
    // all ones but the first pick
    double w[C], sum[NG];
#pragma unroll
    for (int i = 0; i < C; ++i) w[i] = (lane * C + i < n && lane * C + i != node) ? 1.0 : 0.0;
#pragma unroll
    for (int g = 0; g < NG; ++g) sum[g] = 0.0;
    int slot = node % C;
    double us = 0.0;  // lane l: the draw of pick j with j % 32 == l
    // picks after the first node: m - 1 for m >= 2, one for m == 0
    const int picks = (m == 0) ? 1 : m - 1;
#pragma unroll 1
    for (int j = 1; j <= picks; ++j) {
      if (j == 1 || (j & 31) == 0) us = draw((j & ~31) + lane);
      // update_repulsion_choice (maxcut_tfim.py:37-45) for the node picked
      // last, and the sums of the groups that changed (all of them at first)
      uint32_t nz[NW], any[NW];
#pragma unroll
      for (int q = 0; q < NW; ++q) {
        nz[q] = repel ? __ldg(planes + (TABLE ? 2 * plane : 0) + (node * 32 + lane) * NW + q) : 0u;
        any[q] = j == 1 ? 0xFFFFFFFFu
                        : __reduce_or_sync(0xFFFFFFFFu, nz[q]) | ((slot >> 5) == q ? 1u << (slot & 31) : 0u);
      }
      if constexpr (TABLE) {
        const double* row = table + (size_t)node * (32 * C) + 2 * lane;
        if (!repel) {
#pragma unroll
          for (int g = 0; g < NG; ++g) sum[g] = tree_sum<0, SR_GS, SR_GS>(*reinterpret_cast<double(*)[SR_GS]>(&w[SR_GS * g]));
        } else if (sparse) {
#pragma unroll
          for (int g = 0; g < NG; ++g) {
            const uint32_t b = nz[SR_GS * g / 32] >> ((SR_GS * g) & 31);
            if (((any[SR_GS * g / 32] >> ((SR_GS * g) & 31)) & 0xFFu) == 0u) continue;
            double f[SR_GS];
#pragma unroll
            for (int i = 0; i < SR_GS; ++i) {
              f[i] = 1.0;
              if ((b >> i) & 1u) f[i] = __ldg(row + 64 * ((SR_GS * g + i) >> 1) + (i & 1));
            }
#pragma unroll
            for (int i = 0; i < SR_GS; ++i) w[SR_GS * g + i] *= f[i];
            sum[g] = tree_sum<0, SR_GS, SR_GS>(*reinterpret_cast<double(*)[SR_GS]>(&w[SR_GS * g]));
          }
        } else {
#pragma unroll
          for (int g = 0; g < NG; ++g) {
#pragma unroll
            for (int i = 0; i < SR_GS; i += 2) {
              const double2 f = __ldg(reinterpret_cast<const double2*>(row + 32 * (SR_GS * g + i)));
              w[SR_GS * g + i] *= f.x;
              w[SR_GS * g + i + 1] *= f.y;
            }
            sum[g] = tree_sum<0, SR_GS, SR_GS>(*reinterpret_cast<double(*)[SR_GS]>(&w[SR_GS * g]));
          }
        }
      } else {
        uint32_t mm[NW], anym[NW];
#pragma unroll
        for (int q = 0; q < NW; ++q) {
          mm[q] = anym[q] = 0u;
          if (has_minus) {
            mm[q] = repel ? __ldg(planes + plane + (node * 32 + lane) * NW + q) : 0u;
            anym[q] = __reduce_or_sync(0xFFFFFFFFu, mm[q]);
          }
        }
#pragma unroll
        for (int g = 0; g < NG; ++g) {
          const int q = SR_GS * g / 32, sh = (SR_GS * g) & 31;
          if ((((any[q] | anym[q]) >> sh) & 0xFFu) == 0u) continue;
#pragma unroll
          for (int i = 0; i < SR_GS; ++i) mul_if(w[SR_GS * g + i], nz[q] & (1u << (sh + i)), rep1);
          if ((anym[q] >> sh) & 0xFFu) {
#pragma unroll
            for (int i = 0; i < SR_GS; ++i) mul_if(w[SR_GS * g + i], mm[q] & (1u << (sh + i)), repm1);
          }
          sum[g] = tree_sum<0, SR_GS, SR_GS>(*reinterpret_cast<double(*)[SR_GS]>(&w[SR_GS * g]));
        }
      }
      // bit_pick (util:711-724): p = sum(weights) * u, the first node whose
      // running sum is above p; node 0 when none is, or when the roundings of
      // sums in different orders lead to a slot past the last node
      const double loc = tree_sum<0, NG, NG>(sum);
      const double incl = warp_scan(loc);
      const double p = __shfl_sync(0xFFFFFFFFu, incl, 31) * __shfl_sync(0xFFFFFFFFu, us, j & 31);
      const unsigned hit = __ballot_sync(0xFFFFFFFFu, p < incl);
      if (hit) {
        const int owner = __ffs(hit) - 1;
        slot = pick_node<0, C, C>(w, sum, p - (incl - loc), owner, lane);
        node = owner * C + slot;
        if (node >= n) {
          if (lane == 0) w[0] = 0.0;
          slot = node = 0;
        }
      } else {
        if (lane == 0) w[0] = 0.0;
        slot = node = 0;
      }
    }
    // selection mask: weights == 0 (picked, or underflowed to zero); lane l
    // holds bits [l C, l C + C)
    uint64_t bits = 0;
#pragma unroll
    for (int i = 0; i < C; ++i)
      if (lane * C + i < n && w[i] == 0.0) bits |= 1ull << i;
#pragma unroll
    for (int q = 0; q < NW; ++q) {
      // word 32 q + lane: bits from the lane holding its first node on
      const int word = 32 * q + lane, src = 32 * word / C, off = 32 * word - src * C;
      uint64_t v = 0;
#pragma unroll
      for (int t = 0; t * C < 32 + C; ++t) {
        const uint64_t o = __shfl_sync(0xFFFFFFFFu, bits, (src + t) & 31);
        const int at = t * C - off;  // position of that lane's first bit in the word
        if (src + t < 32 && at < 32) v |= at >= 0 ? o << at : o >> -at;
      }
      if (word < n32) out[word] = (uint32_t)v;
    }
  }
}

// Sparse form, n <= 2048 and at most SP_DEG nonzero weights in any row: one
// warp per shot with the weights in shared memory and the sums of groups of 32
// nodes beside them. A pick scans the groups' sums and then one group's weights;
// an update touches the picked node's neighbours, one row slot per lane, and
// sums their groups anew, so a pick costs O(degree) groups instead of n weights.
// The chain of a pick (a row load, the groups' sums, two scans) is latency, so
// what counts is how many shots an SM holds: float64 weights leave 13 at n =
// 2048. Where every weight is +-1 and no row or column has more than SP_CODE_DEG (CODES),
// a weight is one of 2^(SP_CODE_DEG + 1) products of factors in the order of the
// picks, so a byte names it - a leading 1, then a bit per factor; 0 for a picked
// node - and a table holds the products, multiplied in that order.
// Shared memory of one shot: the groups' sums, then the weights or codes of
// 1024 GP nodes. CODES blocks hold the table of products before them.
constexpr int SP_TABLE = 1 << (SP_CODE_DEG + 1);
constexpr int sp_shot_bytes(int GP, bool codes) { return 32 * GP * 8 + 1024 * GP * (codes ? 1 : 8); }
constexpr int sp_warps(bool codes) { return codes ? 4 : 1; }  // shots per block

template <int GP, bool CODES>
__global__ void __launch_bounds__(32 * sp_warps(CODES), CODES ? 12 : 16)
    tfim_sample_sparse_kernel(int n, const double* __restrict__ cum, int ncum, double base, int repel, uint64_t seed,
                              uint64_t round, int shots, uint32_t* __restrict__ theta_out,
                              const SparseEntry* __restrict__ slots, const SampleCtl* __restrict__ ctl, bool codes,
                              bool lists) {
  const SampleCtl ct = *ctl;
  if (sample_form(ct, codes, lists) != (CODES ? SF_CODES : SF_LISTS)) return;
  const int deg = (int)ct.degree;
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31;
  const int n32 = (n + 31) >> 5;  // groups of 32 nodes, and words of a packed row
  double* table = reinterpret_cast<double*>(smem);
  double* gsum = reinterpret_cast<double*>(smem + (CODES ? SP_TABLE * 8 : 0) +
                                           (threadIdx.x >> 5) * sp_shot_bytes(GP, CODES));
  double* w = gsum + 32 * GP;
  uint8_t* code = reinterpret_cast<uint8_t*>(w);
  if constexpr (CODES) {
    const double lnb = log(base);
    const double rep1 = exp(-lnb), repm1 = exp(lnb);
    for (int c = threadIdx.x; c < SP_TABLE; c += blockDim.x) {
      double x = c ? 1.0 : 0.0;
      for (int b = 30 - __clz(c | 1); b >= 0; --b) x *= ((c >> b) & 1) ? repm1 : rep1;
      table[c] = x;
    }
    __syncthreads();
  }
  auto weight = [&](int v) -> double {
    if constexpr (CODES) {
      return table[code[v]];
    } else {
      return w[v];
    }
  };
  const int warps = (gridDim.x * blockDim.x) >> 5;
  for (int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < shots; s += warps) {
    const uint64_t key = mix64(seed ^ mix64(round * 0x632BE59BD9B4E019ull + (uint64_t)s));
    auto draw = [&](int d) {
      const uint64_t h = mix64(key ^ ((uint64_t)d * 0xD1B54A32D192ED03ull));
      return (double)(h >> 11) * (1.0 / 9007199254740992.0);
    };
    const int m = sample_mag(cum, ncum, draw(0));
    int node = s % n;
    uint32_t* out = theta_out + (size_t)s * n32;
    if (m == 1) {
      for (int q = lane; q < n32; q += 32) out[q] = (q == (node >> 5)) ? (1u << (node & 31)) : 0u;
      continue;
    }
    // all ones but the first pick
    for (int v = lane; v < 1024 * GP; v += 32) {
      const bool one = v < n && v != node;
      if constexpr (CODES) {
        code[v] = one ? 1 : 0;
      } else {
        w[v] = one ? 1.0 : 0.0;
      }
    }
    for (int g = lane; g < 32 * GP; g += 32) {
      const int left = n - 32 * g;
      gsum[g] = (double)(left >= 32 ? 32 : left > 0 ? left : 0);
    }
    __syncwarp();
    double us = 0.0;  // lane l: the draw of pick j with j % 32 == l
    const int picks = (m == 0) ? 1 : m - 1;
#pragma unroll 1
    for (int j = 1; j <= picks; ++j) {
      if (j == 1 || (j & 31) == 0) us = draw((j & ~31) + lane);
      // update_repulsion_choice (maxcut_tfim.py:37-45) for the node picked
      // last: lane l its row's slot l (lanes from deg on: the node itself, whose
      // group changed too)
      int col = node;
      if (repel && lane < deg) {
        const SparseEntry e = slots[(size_t)node * SP_DEG + lane];
        col = e.col;
        if constexpr (CODES) {
          const int c = code[col];
          // (a row picked twice, which takes a draw that no prefix is above,
          // could lengthen a full code: left as it is)
          if (c && c < SP_TABLE / 2 && col != node) code[col] = (uint8_t)(2 * c + e.minus);
        } else {
          // (the node itself where the slot is its diagonal, not an empty one: 0
          // stays 0, unless the factor is not finite)
          if (col != node || e.factor != 1.0) w[col] *= e.factor;
        }
      }
      __syncwarp();
      // the touched groups' sums, four at a time by eight lanes each
      const int last = repel ? deg : 0;
#pragma unroll 1
      for (int c = 0; c <= last; c += 4) {
        const int g = __shfl_sync(0xFFFFFFFFu, col, min(c + (lane >> 3), last)) >> 5;
        double x;
        if constexpr (CODES) {
          const uint32_t c4 = *reinterpret_cast<const uint32_t*>(code + 32 * g + 4 * (lane & 7));
          x = (table[c4 & 255u] + table[(c4 >> 8) & 255u]) + (table[(c4 >> 16) & 255u] + table[c4 >> 24]);
        } else {
          const double* wg = w + 32 * g + (lane & 7);
          x = (wg[0] + wg[8]) + (wg[16] + wg[24]);
        }
        x += __shfl_xor_sync(0xFFFFFFFFu, x, 1);
        x += __shfl_xor_sync(0xFFFFFFFFu, x, 2);
        x += __shfl_xor_sync(0xFFFFFFFFu, x, 4);
        if ((lane & 7) == 0) gsum[g] = x;
      }
      __syncwarp();
      // bit_pick (util:711-724): lane l holds the groups GP l .. GP l + GP - 1
      double gs[GP];
#pragma unroll
      for (int i = 0; i < GP; ++i) gs[i] = gsum[GP * lane + i];
      const double loc = tree_sum<0, GP, GP>(gs);
      const double incl = warp_scan(loc);
      const double p = __shfl_sync(0xFFFFFFFFu, incl, 31) * __shfl_sync(0xFFFFFFFFu, us, j & 31);
      const unsigned hit = __ballot_sync(0xFFFFFFFFu, p < incl);
      node = 0;  // no prefix above p
      if (hit) {
        const int owner = __ffs(hit) - 1;
        double q = p - (incl - loc);
        int g = GP * owner;
        if constexpr (GP == 2) {
          const bool up = !(q < gs[0]);
          if (up) q -= gs[0];
          g += (__ballot_sync(0xFFFFFFFFu, up) >> owner) & 1u;
        }
        q = __shfl_sync(0xFFFFFFFFu, q, owner);
        const unsigned h2 = __ballot_sync(0xFFFFFFFFu, q < warp_scan(weight(32 * g + lane)));
        node = 32 * g + (h2 ? __ffs(h2) - 1 : 0);
        node = node < n ? node : 0;  // (led past the last node by a rounding)
      }
      if (lane == 0) {
        if constexpr (CODES) {
          code[node] = 0;
        } else {
          w[node] = 0.0;
        }
      }
      __syncwarp();
    }
    // selection mask: weights == 0 (picked, or underflowed to zero)
    for (int g = 0; g < n32; ++g) {
      const unsigned b = __ballot_sync(0xFFFFFFFFu, 32 * g + lane < n && weight(32 * g + lane) == 0.0);
      if (lane == 0) out[g] = b;
    }
    __syncwarp();
  }
}

// Nonzero counts of W's rows (warp per row).
__global__ void tfim_adj_count_kernel(const float* __restrict__ W, int n, long long* __restrict__ count) {
  const int lane = threadIdx.x & 31;
  for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n; r += (gridDim.x * blockDim.x) >> 5) {
    const float* row = W + (size_t)r * n;
    int c = 0;
    for (int v0 = 0; v0 < n; v0 += 32) {
      const int v = v0 + lane;
      c += __popc(__ballot_sync(0xFFFFFFFFu, v < n && row[v] != 0.0f));
    }
    if (lane == 0) count[r] = c;
  }
}

// Row lists in column order at adj_ptr[r] (warp per row, ballot compaction).
__global__ void tfim_adj_fill_kernel(const float* __restrict__ W, int n,
                                     const long long* __restrict__ adj_ptr, int* __restrict__ adj_col,
                                     float* __restrict__ adj_val) {
  const int lane = threadIdx.x & 31;
  for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n; r += (gridDim.x * blockDim.x) >> 5) {
    const float* row = W + (size_t)r * n;
    long long at = adj_ptr[r];
    for (int v0 = 0; v0 < n; v0 += 32) {
      const int v = v0 + lane;
      const float w = v < n ? row[v] : 0.0f;
      const unsigned nz = __ballot_sync(0xFFFFFFFFu, w != 0.0f);
      if (w != 0.0f) {
        const long long e = at + __popc(nz & ((1u << lane) - 1u));
        adj_col[e] = v;
        adj_val[e] = w;
      }
      at += __popc(nz);
    }
  }
}

}  // namespace pqi

using namespace pqi;

extern "C" {

pqi_status pqi_tfim_jz(const float* W, int n, double* J_eff, unsigned int* degrees,
                       void* workspace, size_t workspace_bytes, void* stream) {
  PQI_CHECK_ARG(W && J_eff && degrees && n > 0);
  Workspace ws(workspace, workspace_bytes);
  float* mn = ws.take<float>(1);
  PQI_CHECK_ARG(mn);
  cudaStream_t s = as_stream(stream);
  PQI_TRY(cudaMemsetAsync(mn, 0xFF, sizeof(float), s));  // max key
  const long long total = (long long)n * n;
  const int g = (int)std::max<long long>(1, std::min<long long>((total + 255) / 256, 148 * 8));
  tfim_min_kernel<<<g, 256, 0, s>>>(W, total, mn);
  PQI_LAUNCHED("tfim_min_kernel");
  tfim_jz_kernel<<<std::max(1, std::min((n + 7) / 8, 148 * 4)), 256, 0, s>>>(W, n, mn, J_eff,
                                                                             degrees);
  PQI_LAUNCHED("tfim_jz_kernel");
  return PQI_OK;
}

pqi_status pqi_tfim_jz_f32(const float* W, int n, double* J_eff, unsigned int* degrees,
                           void* workspace, size_t workspace_bytes, void* stream) {
  PQI_CHECK_ARG(W && J_eff && degrees && n > 0);
  Workspace ws(workspace, workspace_bytes);
  float* mn = ws.take<float>(1);
  PQI_CHECK_ARG(mn);
  cudaStream_t s = as_stream(stream);
  PQI_TRY(cudaMemsetAsync(mn, 0xFF, sizeof(float), s));  // max key
  const long long total = (long long)n * n;
  const int g = (int)std::max<long long>(1, std::min<long long>((total + 255) / 256, 148 * 8));
  tfim_min_kernel<<<g, 256, 0, s>>>(W, total, mn);
  PQI_LAUNCHED("tfim_min_kernel");
  tfim_jz_f32_kernel<<<(n + 127) / 128, 128, 0, s>>>(W, n, mn, J_eff, degrees);
  PQI_LAUNCHED("tfim_jz_f32_kernel");
  return PQI_OK;
}

// Blocks of bins (those below and those above n/2 apart), and slices of the
// pairs: about eight blocks per SM in all.
static int cdf_bin_blocks(int n) {
  return (n / 2 + CDF_BLOCK_BINS) / CDF_BLOCK_BINS + (n - n / 2 + CDF_BLOCK_BINS - 1) / CDF_BLOCK_BINS;
}

static int cdf_slices(int n, long long pairs) {
  const long long bb = cdf_bin_blocks(n), tiles = (pairs + CDF_THREADS / 2 - 1) / (CDF_THREADS / 2);
  return (int)std::max<long long>(1, std::min<long long>(tiles, (148 * 8 + bb - 1) / bb));
}

size_t pqi_tfim_cdf_workspace_bytes(int n, int quality) {
  const long long pairs = (long long)((1 << quality) - 1) * n;
  return (size_t)(cdf_slices(n, pairs) + 1) * (n + 1) * sizeof(double) + 4096;
}

// Whole call at quality 6 (63 steps): n = 1024 82 ms -> 0.48 ms, n = 2048 131 ms
// -> 1.3 ms, against the form that normalised every pair by a pass over its
// n + 1 bins and then summed all pairs in one thread per bin.
pqi_status pqi_tfim_cdf(const double* J_eff, const unsigned int* degrees, int n, int quality,
                        double anneal_t, double anneal_h, const double* thresholds, double* cum,
                        void* workspace, size_t workspace_bytes, void* stream) {
  PQI_CHECK_ARG(J_eff && degrees && thresholds && cum && n >= 3 && quality >= 0 && quality < 30);
  Workspace ws(workspace, workspace_bytes);
  const long long pairs = (long long)((1 << quality) - 1) * n;
  const int slices = cdf_slices(n, pairs);
  double* partial = ws.take<double>((size_t)slices * (n + 1));
  double* hprob = ws.take<double>((size_t)n + 1);
  PQI_CHECK_ARG(partial && hprob);
  cudaStream_t s = as_stream(stream);
  CdfParams P;
  P.n = n;
  P.n_steps = 1 << quality;
  P.tot_t = anneal_t;
  P.delta_t = anneal_t / P.n_steps;
  P.h_mult = fabs(anneal_h);
  P.omega = 1.5 * kPi;
  if (pairs > 0) {
    const long long per = (pairs + slices - 1) / slices;
    tfim_cdf_accum_kernel<<<dim3(cdf_bin_blocks(n), slices), CDF_THREADS, 0, s>>>(P, J_eff, degrees, per, partial);
    PQI_LAUNCHED("tfim_cdf_accum_kernel");
  }
  tfim_cdf_reduce_kernel<<<(n + 32) / 32, 256, 0, s>>>(n, pairs > 0 ? slices : 0, thresholds, partial, hprob);
  PQI_LAUNCHED("tfim_cdf_reduce_kernel");
  tfim_cdf_finish_kernel<<<1, 1024, 0, s>>>(n, hprob, cum);
  PQI_LAUNCHED("tfim_cdf_finish_kernel");
  return PQI_OK;
}

size_t pqi_tfim_sample_workspace_bytes(int n) {
  const int C = (n + 31) / 32;
  // weight tables of the warps (nodes past shared memory), or the register
  // form's row tables (n <= 2048: at most 34 MB, within the former)
  return (size_t)148 * 16 * kWtsPitch * C * sizeof(double) + 4096;
}

static pqi_status tfim_sample_impl(const float* W, int n, const double* cum, double repulsion_base,
                                   uint64_t seed, uint64_t round, int shots, uint32_t* theta_out,
                                   void* workspace, size_t workspace_bytes, void* stream,
                                   const long long* adj_ptr, const int* adj_col, const float* adj_val) {
  // W is read only without row lists (the dense row scan)
  PQI_CHECK_ARG((W || adj_ptr) && cum && theta_out && n >= 3 && shots > 0);
  cudaStream_t s = as_stream(stream);
  const int repel = fabs(1.0 - repulsion_base) <= kEps ? 0 : 1;
  // Up to 2048 nodes with W at hand (and the workspace that
  // pqi_tfim_sample_workspace_bytes names): weights in registers, or the sparse
  // forms - codes from 257 nodes (reg 512: 0.72 ms against 0.80 for 8192 shots),
  // lists from 1025, where the registers hold two warps a scheduler (3-regular
  // 2048: 9.3 ms against 17.0). Milliseconds per round, shared-memory form -> now:
  // ER 1024, 32768 shots 34.9 -> 6.4; ER 2048, 8192 39.7 -> 7.5; complete float
  // 1024, 8192 16.4 -> 2.9; complete float 2000, 4096 49.3 -> 6.9; 3-regular 2048,
  // 16384 19.2 -> 4.3; G(1500, 0.1) float, 8192 12.2 -> 9.4; ER 64, 4096 0.19 -> 0.09.
  if (W && n <= SR_MAX_N) {
    const int RC = ((n + 31) / 32 + SR_GS - 1) / SR_GS * SR_GS, NW = (RC + 31) / 32;
    // codes need factors and their products well inside float64's range
    const bool codes = n > 256 && repulsion_base > 1e-40 && repulsion_base < 1e40;
    const bool lists = n > 1024;
    Workspace ws(workspace, workspace_bytes);
    SampleCtl* ctl = ws.take<SampleCtl>(1);
    uint32_t* planes = ws.take<uint32_t>((size_t)3 * n * 32 * NW);
    double* table = ws.take<double>((size_t)n * 32 * RC);
    SparseEntry* slots = codes || lists ? ws.take<SparseEntry>((size_t)n * SP_DEG) : nullptr;
    if (ctl && planes && table && (slots || !(codes || lists))) {
      // small graphs: one block, which needs no zeroed control words
      const int rb = n <= 256 ? 1 : std::min((n + 3) / 4, 148 * 4), rw = n <= 256 ? 32 : 4;
      if (rb > 1) PQI_TRY(cudaMemsetAsync(ctl, 0, sizeof(SampleCtl), s));
      tfim_rows_kernel<<<rb, 32 * rw, (size_t)rw * 32 * (RC + 1) * sizeof(float), s>>>(W, n, RC, repulsion_base,
                                                                                     planes, table, slots, ctl);
      PQI_LAUNCHED("tfim_rows_kernel");
      auto sparse = [&](auto kern, int GP, bool cd) -> pqi_status {
        const int wb = sp_warps(cd);
        const size_t sm = (size_t)wb * sp_shot_bytes(GP, cd) + (cd ? SP_TABLE * sizeof(double) : 0);
        int per_sm = 1;
        PQI_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
        PQI_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * wb, sm));
        const int g = (int)std::min<long long>(((long long)shots + wb - 1) / wb, 148ll * std::max(1, per_sm));
        kern<<<g, 32 * wb, sm, s>>>(n, cum, n - 1, repulsion_base, repel, seed, round, shots, theta_out, slots, ctl,
                                    codes, lists);
        PQI_LAUNCHED("tfim_sample_sparse_kernel");
        return PQI_OK;
      };
      auto dense = [&](auto kern, int blocks) -> pqi_status {
        const int g = (int)std::min<long long>(((long long)shots + 1) / 2, 148ll * blocks);
        kern<<<g, 64, 0, s>>>(n, cum, n - 1, repulsion_base, repel, seed, round, shots, theta_out, planes, table,
                              ctl, codes, lists);
        PQI_LAUNCHED("tfim_sample_reg_kernel");
        return PQI_OK;
      };
      pqi_status rc = PQI_OK;
      if (codes)
        rc = n <= 1024 ? sparse(tfim_sample_sparse_kernel<1, true>, 1, true)
                       : sparse(tfim_sample_sparse_kernel<2, true>, 2, true);
      if (rc == PQI_OK && lists) rc = sparse(tfim_sample_sparse_kernel<2, false>, 2, false);
      if (rc != PQI_OK) return rc;
#define PQI_SR_CASE(C_)                                                         \
  case C_:                                                                     \
    rc = dense(tfim_sample_reg_kernel<C_, false>, sr_blocks(C_, false));        \
    if (rc == PQI_OK) rc = dense(tfim_sample_reg_kernel<C_, true>, sr_blocks(C_, true)); \
    break
      switch (RC) {
        PQI_SR_CASE(8);
        PQI_SR_CASE(16);
        PQI_SR_CASE(24);
        PQI_SR_CASE(32);
        PQI_SR_CASE(40);
        PQI_SR_CASE(48);
        PQI_SR_CASE(56);
        PQI_SR_CASE(64);
      }
#undef PQI_SR_CASE
      return rc;
    }
  }
  const int C = (n + 31) / 32;
  const size_t per_warp = (size_t)C * kWtsPitch * sizeof(double);
  int wpb = 4;
  size_t smem = per_warp * wpb;
  int use_smem = 1;
  double* wglob = nullptr;
  int grid;
  if (smem <= 160 * 1024) {
    grid = (int)std::min<long long>(((long long)shots + wpb - 1) / wpb, 148 * 8);
    static size_t set_bytes = 0;
    if (smem > 48 * 1024 && smem > set_bytes) {
      PQI_TRY(cudaFuncSetAttribute(tfim_sample_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)smem));
      set_bytes = smem;
    }
  } else {
    use_smem = 0;
    smem = 0;
    Workspace ws(workspace, workspace_bytes);
    const size_t avail = workspace_bytes > 8192 ? workspace_bytes - 8192 : 0;
    const long long warps = std::min<long long>((long long)(avail / per_warp), 148 * 16);
    PQI_CHECK_ARG(warps >= wpb);
    grid = (int)std::min<long long>(warps / wpb, ((long long)shots + wpb - 1) / wpb);
    wglob = ws.take<double>((size_t)grid * wpb * C * kWtsPitch);
    PQI_CHECK_ARG(wglob);
  }
  tfim_sample_kernel<<<grid, 32 * wpb, smem, s>>>(W, n, cum, n - 1, repulsion_base, repel, seed,
                                                   round, shots, theta_out, wglob, use_smem,
                                                   adj_ptr, adj_col, adj_val);
  PQI_LAUNCHED("tfim_sample_kernel");
  return PQI_OK;
}

pqi_status pqi_tfim_sample(const float* W, int n, const double* cum, double repulsion_base,
                           uint64_t seed, uint64_t round, int shots, uint32_t* theta_out,
                           void* workspace, size_t workspace_bytes, void* stream) {
  return tfim_sample_impl(W, n, cum, repulsion_base, seed, round, shots, theta_out, workspace,
                          workspace_bytes, stream, nullptr, nullptr, nullptr);
}

pqi_status pqi_tfim_sample_adj(const float* W, int n, const long long* adj_ptr, const int* adj_col,
                               const float* adj_val, const double* cum, double repulsion_base,
                               uint64_t seed, uint64_t round, int shots, uint32_t* theta_out,
                               void* workspace, size_t workspace_bytes, void* stream) {
  PQI_CHECK_ARG(adj_ptr && (adj_col || !adj_val) && (adj_val || !adj_col));
  return tfim_sample_impl(W, n, cum, repulsion_base, seed, round, shots, theta_out, workspace,
                          workspace_bytes, stream, adj_ptr, adj_col, adj_val);
}

pqi_status pqi_tfim_adj_count(const float* W, int n, long long* count, void* stream) {
  PQI_CHECK_ARG(W && count && n > 0);
  const int blocks = (int)std::min<long long>(((long long)n + 7) / 8, 148 * 16);
  tfim_adj_count_kernel<<<blocks, 256, 0, as_stream(stream)>>>(W, n, count);
  PQI_LAUNCHED("tfim_adj_count_kernel");
  return PQI_OK;
}

pqi_status pqi_tfim_adj_fill(const float* W, int n, const long long* adj_ptr, int* adj_col,
                             float* adj_val, void* stream) {
  PQI_CHECK_ARG(W && adj_ptr && n > 0);
  const int blocks = (int)std::min<long long>(((long long)n + 7) / 8, 148 * 16);
  tfim_adj_fill_kernel<<<blocks, 256, 0, as_stream(stream)>>>(W, n, adj_ptr, adj_col, adj_val);
  PQI_LAUNCHED("tfim_adj_fill_kernel");
  return PQI_OK;
}

}  // extern "C"
