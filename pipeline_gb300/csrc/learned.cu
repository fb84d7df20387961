// Learned CDF of the Morton-key distribution (fit, inference).
//
// Model: a monotone piecewise-linear CDF. Knots x_0 < ... < x_K (x_K = 2^30)
// are distinct keys at evenly spaced ranks of a sorted training sample of keys
// the pipeline produced; heights y_k = (sum_{m<k} softplus(theta_m)) / Z with
// Z = sum_m softplus(theta_m), so 0 = y_0 <= y_1 <= ... <= y_K = 1. A key v in
// segment k maps to F(v) = y_k + (y_{k+1} - y_k) (v - x_k) / (x_{k+1} - x_k).
//
// Fit (all on the GPU): knots from the sorted sample, then Adam steps on
// L = mean_i (F(v_i) - (i + 1/2) / S)^2 with our own forward/backward kernels
// (analytic gradient through the normalised cumulative softplus).
//
// Buckets: exact integer arithmetic on fixed-point tables, so bucket(v) never
// decreases with v and the CPU reference reproduces it bit for bit:
//   Yq_k = round(y_k NB 2^16) (non-decreasing, Yq_0 = 0, Yq_K = NB 2^16),
//   slope_k = floor((Yq_{k+1} - Yq_k) 2^32 / (x_{k+1} - x_k)),
//   bucket(v) = min(NB - 1, (Yq_k + ((v - x_k) slope_k >> 32)) >> 16).
// A 4096-entry table on the top 12 key bits narrows the knot search.
#include "learned.cuh"

namespace octgb {

// ---------------------------------------------------------------- layout --
LcdfLayout lcdf_layout(int max_knots) {
  LcdfLayout L{};
  const size_t K = (size_t)max_knots;  // segments
  size_t o = 256;                      // header
  auto take = [&](size_t bytes) {
    const size_t at = o;
    o = align_up(o + bytes, 256);
    return at;
  };
  L.max_knots = max_knots;
  L.x = take(4 * (K + 1));
  L.theta = take(4 * K);
  L.adam_m = take(4 * K);
  L.adam_v = take(4 * K);
  L.y = take(4 * (K + 1));
  L.g = take(4 * (K + 1));
  L.yq = take(4 * (K + 1));
  L.slope = take(8 * K);
  L.lut = take(2 * (kLcdfLutSize + 1));
  L.bounds = take(4 * ((size_t)kLcdfMaxBuckets + 1));
  L.blut = take(2 * ((size_t)kLcdfBlutSize + 1));
  L.bytes = o;
  return L;
}

__device__ __forceinline__ float softplusf(float t) { return t > 20.f ? t : log1pf(expf(t)); }
__device__ __forceinline__ float sigmoidf_(float t) { return 1.f / (1.f + expf(-t)); }

// Largest k in [lo, hi] with x[k] <= v (x[lo] <= v assumed unless k = lo).
__device__ __forceinline__ int knot_search(const uint32_t* x, int lo, int hi, uint32_t v) {
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (x[mid] <= v) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// ------------------------------------------------------------- knots init --
// One block: knots from the sorted sample; theta = log(e - 1) (softplus 1).
__global__ void __launch_bounds__(1024)
    lcdf_knots_kernel(const uint32_t* __restrict__ sample, int S, int k_req, char* blob,
                      LcdfLayout L) {
  __shared__ uint32_t warp_tot[32];
  __shared__ uint32_t total;
  LcdfHeader* h = reinterpret_cast<LcdfHeader*>(blob);
  uint32_t* x = reinterpret_cast<uint32_t*>(blob + L.x);
  constexpr int PER = (kLcdfMaxKnots + 1023) / 1024;
  uint32_t cand[PER];
  uint32_t keep = 0;
  int cnt = 0;
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int k = threadIdx.x * PER + j;
    cand[j] = 0;
    if (k < k_req) {
      const long long idx = (long long)k * S / k_req;
      cand[j] = sample[idx];
      const uint32_t prev = k == 0 ? 0u : sample[(long long)(k - 1) * S / k_req];
      if (k == 0 || cand[j] != prev) {
        keep |= 1u << j;
        ++cnt;
      }
    }
  }
  uint32_t pos = block_exclusive_sum<1024>((uint32_t)cnt, warp_tot, &total);
#pragma unroll
  for (int j = 0; j < PER; ++j)
    if (keep >> j & 1u) x[pos++] = cand[j];
  const int K = (int)total;
  if (threadIdx.x == 0) {
    x[K] = kLcdfKeyEnd;
    h->magic = kLcdfMagic;
    h->version = kLcdfVersion;
    h->n_knots = K;
    h->max_knots = L.max_knots;
    h->n_sample = S;
    h->steps = 0;
    h->loss = 0.f;
    h->n_buckets = 0;
  }
  float* theta = reinterpret_cast<float*>(blob + L.theta);
  float* m = reinterpret_cast<float*>(blob + L.adam_m);
  float* v = reinterpret_cast<float*>(blob + L.adam_v);
  for (int k = threadIdx.x; k < K; k += 1024) {
    theta[k] = 0.5413248546129181f;  // log(e - 1)
    m[k] = 0.f;
    v[k] = 0.f;
  }
}

// -------------------------------------------------------------- heights --
// One block: y from theta; zero the gradient accumulators and the loss.
__global__ void __launch_bounds__(1024) lcdf_prep_kernel(char* blob, LcdfLayout L) {
  __shared__ float warp_tot[32];
  __shared__ float total;
  LcdfHeader* h = reinterpret_cast<LcdfHeader*>(blob);
  const int K = h->n_knots;
  const float* theta = reinterpret_cast<const float*>(blob + L.theta);
  float* y = reinterpret_cast<float*>(blob + L.y);
  float* g = reinterpret_cast<float*>(blob + L.g);
  constexpr int PER = (kLcdfMaxKnots + 1023) / 1024;
  float s[PER];
  float sum = 0.f;
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int k = threadIdx.x * PER + j;
    s[j] = k < K ? softplusf(theta[k]) : 0.f;
    sum += s[j];
  }
  float run = block_exclusive_sum<1024>(sum, warp_tot, &total);
  const float Z = total;
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int k = threadIdx.x * PER + j;
    if (k < K) y[k] = run / Z;
    run += s[j];
  }
  for (int k = threadIdx.x; k <= K; k += 1024) g[k] = 0.f;
  if (threadIdx.x == 0) {
    y[K] = 1.f;
    h->z = Z;
    h->loss = 0.f;
  }
}

// ------------------------------------------------------ forward/backward --
// One thread per sample key (sorted): loss and dL/dy accumulated per knot.
__global__ void __launch_bounds__(256)
    lcdf_fwd_bwd_kernel(const uint32_t* __restrict__ sample, int S, char* blob, LcdfLayout L) {
  extern __shared__ __align__(16) unsigned char sm[];
  LcdfHeader* h = reinterpret_cast<LcdfHeader*>(blob);
  const int K = h->n_knots;
  uint32_t* sx = reinterpret_cast<uint32_t*>(sm);
  float* sy = reinterpret_cast<float*>(sx + (K + 1));
  float* sg = sy + (K + 1);
  __shared__ float s_loss[8];
  const uint32_t* x = reinterpret_cast<const uint32_t*>(blob + L.x);
  const float* y = reinterpret_cast<const float*>(blob + L.y);
  for (int k = threadIdx.x; k <= K; k += blockDim.x) {
    sx[k] = x[k];
    sy[k] = y[k];
    sg[k] = 0.f;
  }
  __syncthreads();
  float lsum = 0.f;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < S; i += gridDim.x * blockDim.x) {
    const uint32_t v = sample[i];
    int k = 0;
    float f = 0.f;
    if (v >= sx[0]) {
      k = knot_search(sx, 0, K - 1, v);
      f = (float)(v - sx[k]) / (float)(sx[k + 1] - sx[k]);
    }
    const float F = sy[k] + (sy[k + 1] - sy[k]) * f;
    const float t = ((float)i + 0.5f) / (float)S;
    const float r = F - t;
    lsum += r * r;
    const float dF = 2.f * r / (float)S;
    atomicAdd(&sg[k], dF * (1.f - f));
    atomicAdd(&sg[k + 1], dF * f);
  }
  for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
  if ((threadIdx.x & 31) == 0) s_loss[threadIdx.x >> 5] = lsum;
  __syncthreads();
  float* g = reinterpret_cast<float*>(blob + L.g);
  for (int k = threadIdx.x; k <= K; k += blockDim.x)
    if (sg[k] != 0.f) atomicAdd(&g[k], sg[k]);
  if (threadIdx.x == 0) {
    float tot = 0.f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += s_loss[w];
    atomicAdd(&h->loss, tot / (float)S);
  }
}

// --------------------------------------------------------- grad + Adam --
// One block: dL/dtheta_m = sigmoid(theta_m) (sum_{k>m} g_k - sum_k g_k y_k) / Z.
// With grad_out != nullptr the gradient is written out; with lr > 0 one Adam
// step (beta1 0.9, beta2 0.999, eps 1e-8) updates theta.
__global__ void __launch_bounds__(1024)
    lcdf_grad_kernel(char* blob, LcdfLayout L, float* grad_out, float lr) {
  __shared__ float warp_tot[32];
  __shared__ float total;
  __shared__ float red[32];
  LcdfHeader* h = reinterpret_cast<LcdfHeader*>(blob);
  const int K = h->n_knots;
  const float Z = h->z;
  float* theta = reinterpret_cast<float*>(blob + L.theta);
  float* m = reinterpret_cast<float*>(blob + L.adam_m);
  float* v = reinterpret_cast<float*>(blob + L.adam_v);
  const float* y = reinterpret_cast<const float*>(blob + L.y);
  const float* g = reinterpret_cast<const float*>(blob + L.g);
  // gy = sum_k g_k y_k
  float part = 0.f;
  for (int k = threadIdx.x; k <= K; k += 1024) part += g[k] * y[k];
  for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = part;
  __syncthreads();
  if (threadIdx.x < 32) {
    float t = red[threadIdx.x];
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (threadIdx.x == 0) red[0] = t;
  }
  __syncthreads();
  const float gy = red[0];
  // suffix sums over g_1..g_K in reversed blocked order: suf(m+1) = sum_{k>m} g_k
  constexpr int PER = (kLcdfMaxKnots + 1023) / 1024;
  float gv[PER];
  float sum = 0.f;
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int r = threadIdx.x * PER + j;  // r-th from the end: k = K - r
    const int k = K - r;
    gv[j] = (r < K) ? g[k] : 0.f;        // k in [1, K]
    sum += gv[j];
  }
  float run = block_exclusive_sum<1024>(sum, warp_tot, &total);
  const int step = h->steps + 1;
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int r = threadIdx.x * PER + j;
    run += gv[j];  // now sum of g over k in [K - r, K]
    if (r < K) {
      const int mi = K - r - 1;  // theta index: suffix from k = mi + 1
      const float grad = sigmoidf_(theta[mi]) * (run - gy) / Z;
      if (grad_out) grad_out[mi] = grad;
      if (lr > 0.f) {
        const float mm = b1 * m[mi] + (1.f - b1) * grad;
        const float vv = b2 * v[mi] + (1.f - b2) * grad * grad;
        m[mi] = mm;
        v[mi] = vv;
        theta[mi] -= lr * (mm / c1) / (sqrtf(vv / c2) + eps);
      }
    }
  }
  if (threadIdx.x == 0 && lr > 0.f) h->steps = step;
}

// ------------------------------------------------------------ Adam steps --
// All Adam steps of a fit in one launch. The knots stay where they are, so a
// sample key's segment and fraction f never change, and within segment k
//   sum r     = c y'_k + dy_k A          A = sum f, B = sum f^2, C = sum t' f
//   sum r f   = A y'_k + dy_k B - C      (t' and y' from the segment's mean t)
// are all that the gradient needs: five numbers per segment, summed once, in
// place of a pass over the sample (a 12-step search and two shared-memory
// atomics per key) every step. A step is then K independent terms between two
// block-wide scans. Against three launches a step (heights, sample pass,
// gradient) a fit of 100 steps on 262,144 keys and 4,096 segments went from
// 4.2 ms to 0.58 ms (0.38 of it the steps); what bounds it now is the steps' chain of two
// cluster barriers and 64-bit arithmetic, 3.8 us.
// The scans are exact (fixed point in 64 bits: heights in 2^-32, gradients in
// 2^-60), so a fit is the same every time, and closer to 64 bits than sums in
// float: theta 0.8 to 1.7e-6 -> 3.3e-7 off at that size.
struct LcdfMoments {
  float* c;
  float* A;
  float* B;
  float* C;
  uint32_t* mid;  // first + one past last sample rank: twice the mean t times S
  // (of a segment of more than kMomChunk keys A and B hold the first and the one
  // past the last rank, as integers; its sums are those of its parts)
};
static size_t lcdf_moments_bytes() { return 5 * 4 * (size_t)kLcdfMaxSegments; }
static LcdfMoments lcdf_moments_carve(void* base) {
  float* p = static_cast<float*>(base);
  LcdfMoments M;
  M.c = p;
  M.A = p + kLcdfMaxSegments;
  M.B = p + 2 * kLcdfMaxSegments;
  M.C = p + 3 * kLcdfMaxSegments;
  M.mid = reinterpret_cast<uint32_t*>(p + 4 * kLcdfMaxSegments);
  return M;
}

// First rank of the sorted sample whose key is at least v (whole warp: 32
// probes a round, so four dependent loads for 262,144 keys).
__device__ __forceinline__ int warp_lower_rank(const uint32_t* __restrict__ sample, int S,
                                               uint32_t v) {
  const int lane = threadIdx.x & 31;
  long long lo = 0, n = S;  // the answer is in [lo, lo + n]
  while (n > 0) {
    const long long step = (n + 31) / 32;
    const long long at = lo + (long long)(lane + 1) * step - 1;  // last of the lane's part
    const bool below = at < lo + n && sample[at] < v;
    const int parts = __popc(__ballot_sync(0xffffffffu, below));  // whole parts below v
    const long long end = lo + n;
    lo += (long long)parts * step;
    n = min(step - 1, end - lo);  // the next part, without its last key (not below v)
    if (n < 0) n = 0;
  }
  return (int)lo;
}

// A segment of more than kMomChunk keys is summed by chunks of as many ranks
// first, one warp each, so that no warp walks a segment that holds most of the
// sample (one value, or few segments: 2.5 ms for 262,144 keys by one warp, 41 ms
// for 4M, where a stepwise step took 0.04 and 0.34).
constexpr int kMomChunk = 512;
constexpr int kMomRows = kMomChunk / 32;
// The sums of a chunk's first segment and of its last one where that is another,
// ranks counted from the chunk's middle. A segment longer than a chunk is one of
// these in every chunk that it meets.
struct LcdfPart {
  double a, b, c;
};
static size_t lcdf_chunks(int S) { return ((size_t)S + kMomChunk - 1) / kMomChunk; }

template <class T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Segment of key v (whole warp).
__device__ __forceinline__ int warp_segment(const uint32_t* __restrict__ x, int K, uint32_t v) {
  return min(max(warp_lower_rank(x, K, v + 1u) - 1, 0), K - 1);
}

// By the calling warp, in whole numbers (exact, and the 64-bit floating-point pipe
// would bound 4M keys at 0.2 ms); parts of segments that are not longer than a
// chunk are mostly left out (nobody reads them).
__device__ __forceinline__ void lcdf_chunk_parts(const uint32_t* __restrict__ sample, int S,
                                                 const uint32_t* __restrict__ x, int K,
                                                 long long chunk, LcdfPart* __restrict__ parts) {
  const int lane = threadIdx.x & 31;
  const long long r0 = chunk * kMomChunk, r1 = min(r0 + kMomChunk, (long long)S);
  if (r0 >= S) return;
  uint32_t key[kMomRows];
#pragma unroll
  for (int j = 0; j < kMomRows; ++j) {
    const long long i = r0 + j * 32 + lane;
    key[j] = i < r1 ? sample[i] : 0u;
  }
  const uint32_t end = sample[r1 - 1];
  const int s0 = warp_segment(x, K, __shfl_sync(0xffffffffu, key[0], 0));
  const int s1 = s0 == K - 1 || end < x[s0 + 1] ? s0 : warp_segment(x, K, end);
#pragma unroll 1
  for (int slot = 0; slot < 2; ++slot) {
    const int k = slot ? s1 : s0;
    const uint32_t x0 = x[k], x1 = x[k + 1];
    const uint32_t from = k == 0 ? 0u : x0, to = k == K - 1 ? 0xffffffffu : x1;
    int own = 0;  // the segment's keys in this chunk
#pragma unroll
    for (int j = 0; j < kMomRows; ++j)
      own += r0 + j * 32 + lane < r1 && key[j] >= from && (key[j] < to || k == K - 1);
    own = __reduce_add_sync(0xffffffffu, own);
    if (s0 != s1) {  // one end is here: does it reach a chunk's length beyond?
      const long long far = slot ? r1 - own + kMomChunk : r0 + own - kMomChunk - 1;
      if (far < 0 || far >= S) continue;
      const uint32_t v = sample[far];
      if (v < from || (v >= to && k != K - 1)) continue;
    }
    // sums of d, d^2 (its halves apart) and d times twice the rank from the middle
    long long sd = 0, lo = 0, hi = 0, sr = 0;
#pragma unroll
    for (int j = 0; j < kMomRows; ++j) {
      const uint32_t v = key[j];
      if (r0 + j * 32 + lane < r1 && v >= max(from, x0) && (v < to || k == K - 1)) {
        const uint32_t d = v - x0;
        const unsigned long long dd = (unsigned long long)d * d;
        sd += d;
        lo += (uint32_t)dd;
        hi += (uint32_t)(dd >> 32);
        sr += (long long)d * (2 * (j * 32 + lane) + 1 - kMomChunk);
      }
    }
    sd = warp_sum(sd);
    lo = warp_sum(lo);
    hi = warp_sum(hi);
    sr = warp_sum(sr);
    const double inv = 1.0 / (double)(x1 - x0);
    if (lane == 0)
      parts[chunk * 2 + slot] =
          LcdfPart{(double)sd * inv, ((double)hi * 0x1p32 + (double)lo) * inv * inv,
                   (double)sr * inv * (0.5 / (double)S)};
    if (s0 == s1) break;
  }
}

// One warp per segment in the first seg_blocks CTAs, per chunk in the others.
constexpr int kMomWarps = 8;
__global__ void __launch_bounds__(32 * kMomWarps)
    lcdf_moments_kernel(const uint32_t* __restrict__ sample, int S, const char* __restrict__ blob,
                        LcdfLayout L, LcdfMoments M, int k_req, int seg_blocks,
                        LcdfPart* __restrict__ parts) {
  const int K = reinterpret_cast<const LcdfHeader*>(blob)->n_knots;
  const uint32_t* x = reinterpret_cast<const uint32_t*>(blob + L.x);
  const int lane = threadIdx.x & 31, warp = (int)(threadIdx.x >> 5);
  if ((int)blockIdx.x >= seg_blocks) {
    // Knots that are all different lie close: no segment is as long as two
    // steps from one knot's rank to the next.
    if (K == k_req && 2 * (((long long)S + k_req - 1) / k_req) <= kMomChunk) return;
    lcdf_chunk_parts(sample, S, x, K,
                     (long long)((int)blockIdx.x - seg_blocks) * kMomWarps + warp, parts);
    return;
  }
  const int k = (int)blockIdx.x * kMomWarps + warp;
  if (k >= K) return;
  const uint32_t x0 = x[k], x1 = x[k + 1];
  const int a = k == 0 ? 0 : warp_lower_rank(sample, S, x0);
  const int b = k == K - 1 ? S : warp_lower_rank(sample, S, x1);
  if (lane == 0) {
    M.c[k] = (float)(b - a);
    M.mid[k] = (uint32_t)a + (uint32_t)b;
  }
  if (b - a > kMomChunk) {
    if (lane == 0) {
      M.A[k] = __int_as_float(a);
      M.B[k] = __int_as_float(b);
    }
    return;
  }
  const double inv = 1.0 / (double)(x1 - x0), invS = 1.0 / (double)S;
  const double mean = 0.5 * ((double)a + (double)b);
  double sa = 0.0, sb = 0.0, sc = 0.0;
  for (int i = a + lane; i < b; i += 32) {
    const uint32_t v = sample[i];
    const double f = v >= x0 ? (double)(v - x0) * inv : 0.0;  // before the first knot: 0
    sa += f;
    sb += f * f;
    sc += f * (((double)i + 0.5 - mean) * invS);
  }
  sa = warp_sum(sa);
  sb = warp_sum(sb);
  sc = warp_sum(sc);
  if (lane == 0) {
    M.A[k] = (float)sa;
    M.B[k] = (float)sb;
    M.C[k] = (float)sc;
  }
}

// The sums of a segment of ranks [a, b), b - a > kMomChunk, from its parts
// (whole warp).
__device__ __forceinline__ LcdfPart lcdf_long_segment(const LcdfPart* __restrict__ parts, int a,
                                                      int b, int S) {
  const int lane = threadIdx.x & 31;
  const double invS = 1.0 / (double)S, mean = 0.5 * ((double)a + (double)b);
  const int first = a / kMomChunk, last = (b - 1) / kMomChunk;
  LcdfPart s = {0.0, 0.0, 0.0};
#pragma unroll 4
  for (int q = first + lane; q <= last; q += 32) {
    const LcdfPart p = parts[2 * (size_t)q + (q == first && a % kMomChunk != 0 ? 1 : 0)];
    s.a += p.a;
    s.b += p.b;
    s.c += p.c + p.a * (((double)q * kMomChunk + kMomChunk / 2 - mean) * invS);
  }
  return LcdfPart{warp_sum(s.a), warp_sum(s.b), warp_sum(s.c)};
}

// The steps run on one cluster of up to eight CTAs, a segment per thread: one
// CTA took 13 us a step, most of it 64-bit conversions on one SM's pipe.
constexpr int kTrThreads = 512;
constexpr int kTrWarps = kTrThreads / 32;
constexpr int kTrCtas = kLcdfMaxSegments / kTrThreads;
// The fixed point covers heights from 2^-32 to 2^16, i.e. theta above -22;
// theta moves by about lr a step, so fits with steps * lr above this take
// three launches a step instead.
constexpr float kTrMost = 16.f;
static_assert(kTrCtas <= 8, "a portable cluster");

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// v to the same shared-memory place in CTA `rank` of the cluster.
__device__ __forceinline__ void st_cluster(long long* p, uint32_t rank, long long v) {
  uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(a) : "r"(rank));
  asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}

// Warp totals of a cluster-wide scan, in every CTA: one slot per warp.
struct ClusterTotals {
  long long t[kTrCtas * kTrWarps];
};

// Inclusive scan within the warp; its total to every CTA's table.
__device__ __forceinline__ long long cluster_scan_send(long long v, ClusterTotals& T) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  long long inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  const long long total = __shfl_sync(0xffffffffu, inc, 31);
  if (lane < (int)gridDim.x) st_cluster(&T.t[blockIdx.x * kTrWarps + w], (uint32_t)lane, total);
  return inc;
}
// After the cluster barrier: the sum of the warps before this one, and of all.
__device__ __forceinline__ long long cluster_scan_read(const ClusterTotals& T, long long& total) {
  const int lane = threadIdx.x & 31;
  const int me = blockIdx.x * kTrWarps + (int)(threadIdx.x >> 5);
  const int n = (int)gridDim.x * kTrWarps;
  long long before = 0, all = 0;
#pragma unroll
  for (int j = 0; j < kTrCtas * kTrWarps / 32; ++j) {
    const int i = j * 32 + lane;
    const long long t = i < n ? T.t[i] : 0;
    all += t;
    before += i < me ? t : 0;
  }
  total = warp_sum(all);
  return warp_sum(before);
}

__global__ void __launch_bounds__(kTrThreads)
    lcdf_train_kernel(char* blob, LcdfLayout L, LcdfMoments M, const LcdfPart* parts, int S,
                      int steps, float lr) {
  // three tables a step; each is written again only after a barrier that
  // follows its last read
  __shared__ ClusterTotals s_height, s_grad, s_gy;
  LcdfHeader* h = reinterpret_cast<LcdfHeader*>(blob);
  const int K = h->n_knots, step0 = h->steps;
  const int k = (int)(blockIdx.x * kTrThreads + threadIdx.x), lane = threadIdx.x & 31;
  const bool in = k < K;
  float* g_theta = reinterpret_cast<float*>(blob + L.theta);
  float* g_m = reinterpret_cast<float*>(blob + L.adam_m);
  float* g_v = reinterpret_cast<float*>(blob + L.adam_v);
  const float c = in ? M.c[k] : 0.f;
  float A = in ? M.A[k] : 0.f, B = in ? M.B[k] : 0.f, C = in ? M.C[k] : 0.f;
  for (uint32_t todo = __ballot_sync(0xffffffffu, c > (float)kMomChunk); todo; todo &= todo - 1u) {
    const int src = __ffs(todo) - 1;  // a lane's segment is long: the warp adds its parts
    const LcdfPart p = lcdf_long_segment(parts, __shfl_sync(0xffffffffu, __float_as_int(A), src),
                                         __shfl_sync(0xffffffffu, __float_as_int(B), src), S);
    if (lane == src) {
      A = (float)p.a;
      B = (float)p.b;
      C = (float)p.c;
    }
  }
  const unsigned long long mid = in ? M.mid[k] : 0u;
  float th = in ? g_theta[k] : 0.f, m = in ? g_m[k] : 0.f, v = in ? g_v[k] : 0.f;
  const unsigned long long two_s = 2ull * (unsigned)S;
  const float w = 2.f / (float)S, inv2s = 0.5f / (float)S;
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  cluster_barrier();  // every CTA's tables exist
  for (int it = 0; it < steps; ++it) {
    const float s = in ? softplusf(th) : 0.f;
    const long long fix = __float2ll_rn(s * 0x1p32f);
    const long long inc = cluster_scan_send(fix, s_height);
    cluster_barrier();
    long long Z;
    const long long cum = cluster_scan_read(s_height, Z) + inc - fix;
    Z = max(Z, 1ll);
    // mid / (2 S) of Z: whole parts and the rest's share
    const unsigned long long q = (unsigned long long)Z / two_s;
    const unsigned long long rem = (unsigned long long)Z - q * two_s;
    const float invz = 1.f / (float)Z;  // of fixed-point values
    const float inv_height = 1.f / ((float)Z * 0x1p-32f);
    const long long at_mean = (long long)(mid * q) + __float2ll_rn((float)(mid * rem) * inv2s);
    const float yp = (float)(cum - at_mean) * invz;
    const float dy = s * inv_height;
    const float sr = c * yp + dy * A;
    const float srf = A * yp + dy * B - C;
    const float a0 = w * (sr - srf), a1 = w * srf;
    const long long g0 = __float2ll_rn(a0 * 0x1p60f), g1 = __float2ll_rn(a1 * 0x1p60f);
    const float y0 = (float)cum * invz, y1 = (float)(cum + fix) * invz;
    const long long gy_own =
        __float2ll_rn(a0 * y0 * 0x1p60f) + __float2ll_rn(a1 * y1 * 0x1p60f);
    const long long ginc = cluster_scan_send(g0 + g1, s_grad);
    const long long gy_warp = warp_sum(gy_own);
    if (lane < (int)gridDim.x)
      st_cluster(&s_gy.t[blockIdx.x * kTrWarps + (threadIdx.x >> 5)], (uint32_t)lane, gy_warp);
    const int step = step0 + it + 1;
    const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
    const float sig = sigmoidf_(th) * inv_height;
    cluster_barrier();
    long long T, gy;
    const long long E = cluster_scan_read(s_grad, T) + ginc - (g0 + g1);
    cluster_scan_read(s_gy, gy);
    // sum of g over knots k + 1 on: everything but the knots up to k's share of k
    const long long after = T - E - g0;
    const float grad = sig * ((float)(after - gy) * 0x1p-60f);
    m = b1 * m + (1.f - b1) * grad;
    v = b2 * v + (1.f - b2) * grad * grad;
    th -= lr * (m / c1) / (sqrtf(v / c2) + eps);
  }
  if (in) {
    g_theta[k] = th;
    g_m[k] = m;
    g_v[k] = v;
  }
  // (every CTA has read the header: the barriers above)
  if (k == 0) h->steps = step0 + steps;
}

// ------------------------------------------------------ fixed-point tables --
// One block: Yq, slopes and the top-bits lookup table for NB buckets.
__global__ void __launch_bounds__(1024) lcdf_tables_kernel(char* blob, LcdfLayout L, int nb) {
  __shared__ uint32_t warp_tot[32];
  LcdfHeader* h = reinterpret_cast<LcdfHeader*>(blob);
  const int K = h->n_knots;
  const uint32_t* x = reinterpret_cast<const uint32_t*>(blob + L.x);
  const float* y = reinterpret_cast<const float*>(blob + L.y);
  uint32_t* yq = reinterpret_cast<uint32_t*>(blob + L.yq);
  unsigned long long* slope = reinterpret_cast<unsigned long long*>(blob + L.slope);
  uint16_t* lut = reinterpret_cast<uint16_t*>(blob + L.lut);
  const uint32_t top = (uint32_t)nb << kLcdfFix;
  // Yq_k = round(y_k * NB * 2^16), then a running max keeps it non-decreasing.
  constexpr int PER = (kLcdfMaxKnots + 1023) / 1024;
  uint32_t q[PER];
  uint32_t mx = 0;
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int k = threadIdx.x * PER + j;
    q[j] = 0;
    if (k <= K) {
      double t = (double)y[k] * (double)top;
      uint32_t u = (uint32_t)min((double)top, max(0.0, rint(t)));
      if (k == 0) u = 0;
      if (k == K) u = top;
      q[j] = u;
    }
    mx = max(mx, q[j]);
    q[j] = mx;  // running max within the thread's block
  }
  // exclusive max-scan across threads
  uint32_t inc = mx;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc = max(inc, t);
  }
  if (lane == 31) warp_tot[w] = inc;
  __syncthreads();
  if (w == 0) {
    uint32_t t = warp_tot[lane];
    uint32_t ti = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(0xffffffffu, ti, o);
      if (lane >= o) ti = max(ti, u);
    }
    warp_tot[lane] = ti;  // inclusive max of warps 0..lane
  }
  __syncthreads();
  uint32_t before = __shfl_up_sync(0xffffffffu, inc, 1);
  if (lane == 0) before = 0;
  if (w > 0) before = max(before, warp_tot[w - 1]);
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int k = threadIdx.x * PER + j;
    if (k <= K) yq[k] = max(before, q[j]);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < K; k += 1024) {
    const unsigned long long dy = (unsigned long long)(yq[k + 1] - yq[k]);
    slope[k] = (dy << 32) / (unsigned long long)(x[k + 1] - x[k]);
  }
  // lut[p] = number of knots x_k (k < K) with x_k <= p << 18, for p in [0, 4096].
  for (int p = threadIdx.x; p <= kLcdfLutSize; p += 1024) {
    const uint32_t v = (uint32_t)p << (30 - kLcdfLutBits);
    int lo = 0, hi = K;  // count of x[0..K) <= v
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (x[mid] <= v) lo = mid + 1;
      else hi = mid;
    }
    lut[p] = (uint16_t)lo;
  }
  if (threadIdx.x == 0) h->n_buckets = nb;
}

// Bucket boundaries of the fixed-point model, for the bucketed sort:
// bounds[b] = smallest key v with bucket(v) >= b (bounds[0] = 0; 2^30 when no
// key reaches b; bounds[nb] = 2^30), and blut[p] = bucket(p << 16) for the
// 2^14 cells of 2^16 keys (blut[2^14] = bucket(2^30 - 1)). Because bucket()
// never decreases, bucket(v) = the largest b with bounds[b] <= v, and that b
// lies in [blut[v >> 16], blut[(v >> 16) + 1]].
__global__ void __launch_bounds__(256) lcdf_bounds_kernel(char* blob, LcdfLayout L, int nb) {
  const LcdfTables t = lcdf_tables_global(blob, L);
  uint32_t* bounds = reinterpret_cast<uint32_t*>(blob + L.bounds);
  uint16_t* blut = reinterpret_cast<uint16_t*>(blob + L.blut);
  const int items = nb + 1 + kLcdfBlutSize + 1;
  for (int it = blockIdx.x * blockDim.x + threadIdx.x; it < items; it += gridDim.x * blockDim.x) {
    if (it <= nb) {
      const uint32_t b = (uint32_t)it;
      uint32_t v;
      if (b == 0) {
        v = 0;
      } else if (b == (uint32_t)nb || lcdf_bucket(t, kLcdfKeyEnd - 1u) < b) {
        v = kLcdfKeyEnd;
      } else {
        uint32_t lo = 0, hi = kLcdfKeyEnd - 1u;  // bucket(hi) >= b
        while (lo < hi) {
          const uint32_t mid = lo + ((hi - lo) >> 1);
          if (lcdf_bucket(t, mid) >= b) hi = mid;
          else lo = mid + 1;
        }
        v = lo;
      }
      bounds[b] = v;
    } else {
      const int p = it - (nb + 1);
      const uint32_t v = min((uint32_t)p << (30 - kLcdfBlutBits), kLcdfKeyEnd - 1u);
      blut[p] = (uint16_t)lcdf_bucket(t, v);
    }
  }
}

static void launch_lcdf_bounds(char* blob, const LcdfLayout& L, int nb, cudaStream_t s) {
  const int items = nb + 1 + kLcdfBlutSize + 1;
  lcdf_bounds_kernel<<<(items + 255) / 256, 256, 0, s>>>(blob, L, nb);
}

// ------------------------------------------------------------- inference --
__global__ void __launch_bounds__(256)
    lcdf_bucket_kernel(const char* __restrict__ blob, LcdfLayout L, const uint32_t* __restrict__ keys,
                       int n, uint32_t* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char sm[];
  LcdfTables t = lcdf_load_tables(blob, L, sm);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    out[i] = lcdf_bucket(t, keys[i]);
}

size_t lcdf_tables_smem(int max_knots) {
  return align_up(8 * (size_t)max_knots + 4 * (size_t)(max_knots + 1) * 2 +
                      2 * (kLcdfLutSize + 1),
                  16);
}

cudaError_t launch_lcdf_train(const uint32_t* sorted_sample, int S, int steps, float lr, char* blob,
                              const LcdfLayout& L, cudaStream_t s) {
  const size_t fb_smem = 12 * (size_t)(L.max_knots + 1);
  set_smem_limit(lcdf_fwd_bwd_kernel, 12 * (kLcdfMaxSegments + 1));
  int grid = (S + 255) / 256;
  if (grid > device_sm_count() * 4) grid = device_sm_count() * 4;
  if (grid < 1) grid = 1;
  for (int it = 0; it < steps; ++it) {
    lcdf_prep_kernel<<<1, 1024, 0, s>>>(blob, L);
    lcdf_fwd_bwd_kernel<<<grid, 256, fb_smem, s>>>(sorted_sample, S, blob, L);
    lcdf_grad_kernel<<<1, 1024, 0, s>>>(blob, L, nullptr, lr);
  }
  return cudaGetLastError();
}

cudaError_t launch_lcdf_fit(const uint32_t* sorted_sample, int S, int k_req, int steps, float lr,
                            char* blob, const LcdfLayout& L, int nb, void* moments, void* scratch,
                            cudaStream_t s) {
  lcdf_knots_kernel<<<1, 1024, 0, s>>>(sorted_sample, S, k_req, blob, L);
  const size_t fb_smem = 12 * (size_t)(L.max_knots + 1);
  int grid = (S + 255) / 256;
  if (grid > device_sm_count() * 4) grid = device_sm_count() * 4;
  if (grid < 1) grid = 1;
  set_smem_limit(lcdf_fwd_bwd_kernel, 12 * (kLcdfMaxSegments + 1));
  // (a rate that is not positive moves nothing, as in the stepwise kernels)
  if (steps > 0 && lr > 0.f && (float)steps * lr <= kTrMost) {
    const LcdfMoments M = lcdf_moments_carve(moments);
    LcdfPart* parts = static_cast<LcdfPart*>(scratch);
    const int seg_blocks = (k_req + kMomWarps - 1) / kMomWarps;
    const size_t chunks = S > kMomChunk ? lcdf_chunks(S) : 0;  // (fewer keys: no long segment)
    const unsigned blocks = seg_blocks + (unsigned)((chunks + kMomWarps - 1) / kMomWarps);
    lcdf_moments_kernel<<<blocks, 32 * kMomWarps, 0, s>>>(sorted_sample, S, blob, L, M, k_req,
                                                          seg_blocks, parts);
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3((k_req + kTrThreads - 1) / kTrThreads);
    c.blockDim = dim3(kTrThreads);
    c.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {c.gridDim.x, 1u, 1u};
    c.attrs = at;
    c.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&c, lcdf_train_kernel, blob, L, M, parts, S, steps, lr);
    if (e != cudaSuccess) return e;
  } else {  // heights could leave the fixed point's range, or nothing moves
    const cudaError_t e = launch_lcdf_train(sorted_sample, S, steps, lr, blob, L, s);
    if (e != cudaSuccess) return e;
  }
  // final heights, loss of the trained model, tables
  lcdf_prep_kernel<<<1, 1024, 0, s>>>(blob, L);
  lcdf_fwd_bwd_kernel<<<grid, 256, fb_smem, s>>>(sorted_sample, S, blob, L);
  lcdf_tables_kernel<<<1, 1024, 0, s>>>(blob, L, nb);
  launch_lcdf_bounds(blob, L, nb, s);
  return cudaGetLastError();
}

cudaError_t launch_lcdf_loss_grad(const uint32_t* sorted_sample, int S, char* blob,
                                  const LcdfLayout& L, float* grad_out, cudaStream_t s) {
  const size_t fb_smem = 12 * (size_t)(L.max_knots + 1);
  set_smem_limit(lcdf_fwd_bwd_kernel, 12 * (kLcdfMaxSegments + 1));
  int grid = (S + 255) / 256;
  if (grid > device_sm_count() * 4) grid = device_sm_count() * 4;
  if (grid < 1) grid = 1;
  lcdf_prep_kernel<<<1, 1024, 0, s>>>(blob, L);
  lcdf_fwd_bwd_kernel<<<grid, 256, fb_smem, s>>>(sorted_sample, S, blob, L);
  lcdf_grad_kernel<<<1, 1024, 0, s>>>(blob, L, grad_out, 0.f);
  return cudaGetLastError();
}

cudaError_t launch_lcdf_tables(char* blob, const LcdfLayout& L, int nb, cudaStream_t s) {
  lcdf_prep_kernel<<<1, 1024, 0, s>>>(blob, L);
  lcdf_tables_kernel<<<1, 1024, 0, s>>>(blob, L, nb);
  launch_lcdf_bounds(blob, L, nb, s);
  return cudaGetLastError();
}

cudaError_t launch_lcdf_buckets(const char* blob, const LcdfLayout& L, const uint32_t* keys, int n,
                                uint32_t* out, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const size_t smem = lcdf_tables_smem(L.max_knots);
  set_smem_limit(lcdf_bucket_kernel, (int)lcdf_tables_smem(kLcdfMaxSegments));
  int grid = (n + 255) / 256;
  if (grid > device_sm_count() * 8) grid = device_sm_count() * 8;
  lcdf_bucket_kernel<<<grid, 256, smem, s>>>(blob, L, keys, n, out);
  return cudaGetLastError();
}

}  // namespace octgb

// ------------------------------------------------------------------ C ABI --
extern "C" {

OCT_API int oct_lcdf_layout(int max_segments, size_t offsets[12]) {
  using namespace octgb;
  if (max_segments < 1 || max_segments > kLcdfMaxSegments || !offsets) return OCT_ERR_INVALID_ARG;
  const LcdfLayout L = lcdf_layout(max_segments);
  const size_t v[12] = {L.x,   L.theta, L.adam_m, L.adam_v, L.y,    L.g,
                        L.yq,  L.slope, L.lut,    L.bounds, L.blut, L.bytes};
  for (int i = 0; i < 12; ++i) offsets[i] = v[i];
  return OCT_OK;
}

OCT_API size_t oct_lcdf_fit_workspace_bytes(int n_sample) {
  using namespace octgb;
  if (n_sample < 1) return 0;
  return align_up(sort_keys_bytes(n_sample, 30), 256) + 2 * align_up(4 * (size_t)n_sample, 256) +
         lcdf_moments_bytes();
}

OCT_API int oct_lcdf_fit(const uint32_t* sample_keys, int n_sample, int n_segments, int steps,
                         float lr, int n_buckets, void* model, int max_segments, void* workspace,
                         size_t workspace_bytes, oct_stream_t stream) {
  using namespace octgb;
  if (!sample_keys || !model || !workspace || n_sample < 1 || n_sample > OCT_MAX_N ||
      n_segments < 1 || n_segments > max_segments || max_segments > kLcdfMaxSegments ||
      steps < 0 || n_buckets < 1 || n_buckets > kLcdfMaxBuckets || (reinterpret_cast<uintptr_t>(workspace) & 255))
    return OCT_ERR_INVALID_ARG;
  if (workspace_bytes < oct_lcdf_fit_workspace_bytes(n_sample)) return OCT_ERR_WORKSPACE;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  char* w = static_cast<char*>(workspace);
  uint32_t* keys = reinterpret_cast<uint32_t*>(w + align_up(sort_keys_bytes(n_sample, 30), 256));
  uint32_t* alt = keys + align_up(4 * (size_t)n_sample, 256) / 4;
  cudaError_t e = cudaMemcpyAsync(keys, sample_keys, 4 * (size_t)n_sample, cudaMemcpyDeviceToDevice, s);
  if (e == cudaSuccess && n_sample > 1)
    e = launch_sort_keys(keys, alt, n_sample, 30, w, nullptr, s);
  const LcdfLayout L = lcdf_layout(max_segments);
  if (e == cudaSuccess)
    e = launch_lcdf_fit(keys, n_sample, n_segments, steps, lr, static_cast<char*>(model), L,
                        n_buckets, alt + align_up(4 * (size_t)n_sample, 256) / 4, alt, s);
  if (e != cudaSuccess) {
    set_last_error(cudaGetErrorString(e));
    return OCT_ERR_CUDA;
  }
  return OCT_OK;
}

OCT_API int oct_lcdf_loss_grad(const uint32_t* sorted_sample, int n_sample, void* model,
                               int max_segments, float* d_grad, oct_stream_t stream) {
  using namespace octgb;
  if (!sorted_sample || !model || n_sample < 1 || max_segments < 1 ||
      max_segments > kLcdfMaxSegments)
    return OCT_ERR_INVALID_ARG;
  const LcdfLayout L = lcdf_layout(max_segments);
  cudaError_t e = launch_lcdf_loss_grad(sorted_sample, n_sample, static_cast<char*>(model), L,
                                        d_grad, reinterpret_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) {
    set_last_error(cudaGetErrorString(e));
    return OCT_ERR_CUDA;
  }
  return OCT_OK;
}

OCT_API int oct_lcdf_tables(void* model, int max_segments, int n_buckets, oct_stream_t stream) {
  using namespace octgb;
  if (!model || max_segments < 1 || max_segments > kLcdfMaxSegments || n_buckets < 1 ||
      n_buckets > kLcdfMaxBuckets)
    return OCT_ERR_INVALID_ARG;
  const LcdfLayout L = lcdf_layout(max_segments);
  cudaError_t e = launch_lcdf_tables(static_cast<char*>(model), L, n_buckets,
                                     reinterpret_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) {
    set_last_error(cudaGetErrorString(e));
    return OCT_ERR_CUDA;
  }
  return OCT_OK;
}

OCT_API int oct_lcdf_buckets(const void* model, int max_segments, const uint32_t* keys, int n,
                             uint32_t* d_buckets, oct_stream_t stream) {
  using namespace octgb;
  if (!model || n < 0 || max_segments < 1 || max_segments > kLcdfMaxSegments) return OCT_ERR_INVALID_ARG;
  if (n == 0) return OCT_OK;
  if (!keys || !d_buckets) return OCT_ERR_INVALID_ARG;
  const LcdfLayout L = lcdf_layout(max_segments);
  cudaError_t e = launch_lcdf_buckets(static_cast<const char*>(model), L, keys, n, d_buckets,
                                      reinterpret_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) {
    set_last_error(cudaGetErrorString(e));
    return OCT_ERR_CUDA;
  }
  return OCT_OK;
}

}  // extern "C"

extern "C" {

// `steps` further Adam steps on the model's current parameters (sorted sample).
OCT_API int oct_lcdf_train_steps(const uint32_t* sorted_sample, int n_sample, void* model,
                                 int max_segments, int steps, float lr, oct_stream_t stream) {
  using namespace octgb;
  if (!sorted_sample || !model || n_sample < 1 || steps < 0 || max_segments < 1 ||
      max_segments > kLcdfMaxSegments || !(lr > 0.f))
    return OCT_ERR_INVALID_ARG;
  const LcdfLayout L = lcdf_layout(max_segments);
  cudaError_t e = launch_lcdf_train(sorted_sample, n_sample, steps, lr, static_cast<char*>(model),
                                    L, reinterpret_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) {
    set_last_error(cudaGetErrorString(e));
    return OCT_ERR_CUDA;
  }
  return OCT_OK;
}

}  // extern "C"
