// Delta rules over packed batches, sixteen tokens at a time (see vector_delta.cu), g one number per head or a vector
// over its key channels:
//
//   S <- diag(g) S;  u = beta (v - S^T k);  S <- S + k u^T;  o = S^T q
//
// With S0 the state before a chunk of sixteen tokens, P_t = g_1 .. g_t and R_it = g_(i+1) .. g_t, the writes u_t solve
// (I + L) U = beta (V - (P K) S0), L_ti = beta_t k_t . (R_it k_i) for i < t, so with M = (I + L)^-1 diag(beta)
//
//   U = M (V - (P K) S0);   O = (P Q) S0 + W U, W_ti = q_t . (R_it k_i) for i <= t;   S' = P_16 S0 + (R_t16 K)^T U
//
//   head_gram_kernel, channel_gram_kernel    M and W of every chunk and head (and the decays of a head)
//   chunk_delta_kernel                       the recurrence
//
// No quotient of decays is formed: a product over a span is taken factor by factor, so nothing overflows.
//
// The chain from chunk to chunk is three small products.  They run on the tensor cores with FP32 operands split into
// two TF32 parts each and three products (22 bits of a product; sums in FP32).  Token by token, or four tokens at a
// time on the FP32 units, a chunk's sixteen tokens took sixteen or four rounds of shuffles and dependent sums.
// mma.sync and not tcgen05: a chunk's operands come from registers (the state's accumulators are the next product's A
// operand as they stand, its channels merely taken in another order), and a round through tensor memory costs
// more than these products do.
//
// A CTA owns 32 value columns of one head of one sequence: two tiles of sixteen columns, each two warps that share
// the channels.  A warp holds S^T [16 columns, D / 2 channels] as accumulators.  Partial K S0 and Q S0 meet in shared
// memory; both warps of a tile solve U.  The vectors of the next chunks are fetched into a ring in shared memory; with a
// decay per channel they are multiplied with their decays there, a chunk ahead.  A sequence whose first packed row
// stands at position 0 starts from a zero state whatever its slot holds; a negative slot marks padding.
#include "include/us_common.cuh"

namespace {

constexpr int kChunk = 16;        // tokens whose products share a state
constexpr int kCols = 32;         // value columns per CTA
constexpr int kSplit = 2;         // warps that share a tile's channels
constexpr int kTiles = kCols / 16;
constexpr int kThreads = 32 * kSplit * kTiles;
constexpr int kBufs = 3;          // chunks in shared memory
constexpr int kMaxDim = 256;

// Coefficients of a chunk and head: M [t][i] | W [t][i] | with a decay per head P_t | R_t16
constexpr int kM = 0, kW = 256, kP = 512, kR = 528, kCoef = 544;

struct DeltaRule {
  const float *q, *k, *v;         // [rows, Hk, D] x 2, [rows, H, V]
  const float *g, *beta;          // [rows, H] or [rows, H, D], [rows, H]
  float* coef;                    // [rows / 16 + B, H, kCoef]
  float* state;                   // [slots, H, D, V]
  float* out;                     // [rows, H, V]
  const int *cu, *slots, *pos;
  int B, H, Hk, D, V;
};

// first chunk of sequence s among all of a batch's (one of at least a sixteenth of its rows each)
__device__ __forceinline__ long long first_chunk(int start, int s) { return (start >> 4) + s; }

// sequence, its first row and length, and the chunk in it, of a batch's `chunk`-th one; false past the last
__device__ __forceinline__ bool find_chunk(const DeltaRule& a, int& s, int& start, int& n, int& chunk) {
  for (s = 0; s < a.B; ++s) {
    start = a.cu[s];
    n = a.cu[s + 1] - start;
    const int chunks = (n + kChunk - 1) / kChunk;
    if (chunk < chunks) return a.slots[s] >= 0;
    chunk -= chunks;
  }
  return false;
}

// M from L (strictly lower) and beta: column `lane` by forward substitution.
__device__ __forceinline__ void solve_columns(const float (*low)[kChunk + 1], const float* beta, float* out, int lane) {
  if (lane >= kChunk) return;
  float m[kChunk];
#pragma unroll
  for (int x = 0; x < kChunk; ++x) {
    float sum = x == lane ? beta[x] : 0.f;
#pragma unroll
    for (int y = 0; y < x; ++y) sum = fmaf(-low[x][y], m[y], sum);
    m[x] = sum;
    out[kM + x * kChunk + lane] = sum;
  }
}

constexpr int kGramWarps = 4, kGramPitch = 36;   // 32 channels at a time, rows apart by 4 banks

// A warp per key head of a chunk: lane = (token t, half of the tokens i).
__global__ void __launch_bounds__(kGramWarps * 32) head_gram_kernel(const DeltaRule a) {
  US_PDL_PROLOGUE();
  __shared__ __align__(16) float rows_[kGramWarps][2 * kChunk * kGramPitch];
  __shared__ float low[kGramWarps][kChunk][kChunk + 1], decay[kGramWarps][2][kChunk];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int s, start, n, chunk = blockIdx.x;
  const int hk = blockIdx.y * kGramWarps + warp;
  if (!find_chunk(a, s, start, n, chunk) || hk >= a.Hk) return;
  const long long row = start + (long long)chunk * kChunk;
  const int rows = min(kChunk, n - chunk * kChunk), rep = a.H / a.Hk;
  float* kr = rows_[warp];
  float* qr = kr + kChunk * kGramPitch;
  const int t = lane >> 1, i0 = (lane & 1) * 8;
  float kk[8], qk[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) kk[e] = qk[e] = 0.f;
  for (int c0 = 0; c0 < a.D; c0 += 32) {
    __syncwarp();
    const int c = c0 + lane;
#pragma unroll
    for (int e = 0; e < kChunk; ++e) {
      const long long at = ((row + e) * a.Hk + hk) * a.D + c;
      const bool in = e < rows && c < a.D;
      kr[e * kGramPitch + lane] = in ? a.k[at] : 0.f;
      qr[e * kGramPitch + lane] = in ? a.q[at] : 0.f;
    }
    __syncwarp();
#pragma unroll
    for (int d = 0; d < 32; d += 4) {
      const float4 kt = *reinterpret_cast<const float4*>(kr + t * kGramPitch + d);
      const float4 qt = *reinterpret_cast<const float4*>(qr + t * kGramPitch + d);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float4 ki = *reinterpret_cast<const float4*>(kr + (i0 + e) * kGramPitch + d);
        kk[e] = fmaf(kt.x, ki.x, fmaf(kt.y, ki.y, fmaf(kt.z, ki.z, fmaf(kt.w, ki.w, kk[e]))));
        qk[e] = fmaf(qt.x, ki.x, fmaf(qt.y, ki.y, fmaf(qt.z, ki.z, fmaf(qt.w, ki.w, qk[e]))));
      }
    }
  }
  for (int h = hk * rep; h < (hk + 1) * rep; ++h) {
    float* out = a.coef + ((first_chunk(start, s) + chunk) * a.H + h) * kCoef;
    __syncwarp();
    if (lane < kChunk) {
      decay[warp][0][lane] = lane < rows ? a.g[(row + lane) * a.H + h] : 1.f;
      decay[warp][1][lane] = lane < rows ? a.beta[(row + lane) * a.H + h] : 0.f;
    }
    __syncwarp();
    const float* g = decay[warp][0];
    const float beta_t = decay[warp][1][t];
    float r = 1.f;                                   // g_(i+1) .. g_t, from i = t down to this lane's tokens
    for (int i = t - 1; i >= i0 + 8; --i) r *= g[i + 1];
#pragma unroll
    for (int e = 7; e >= 0; --e) {
      const int i = i0 + e;
      if (i < t) r *= g[i + 1];
      low[warp][t][i] = i < t ? beta_t * r * kk[e] : 0.f;
      out[kW + t * kChunk + i] = i <= t ? r * qk[e] : 0.f;
    }
    if (lane < kChunk) {
      float p = 1.f, tail = 1.f;
      for (int x = 0; x <= lane; ++x) p *= g[x];
      for (int x = lane + 1; x < kChunk; ++x) tail *= g[x];
      out[kP + lane] = p;
      out[kR + lane] = tail;
    }
    __syncwarp();
    solve_columns(low[warp], decay[warp][1], out, lane);
  }
}

// Four neighbouring channels, zeros (or `rest`) past the width.
__device__ __forceinline__ float4 load_four(const float* p, int d, int D, bool quad, float rest) {
  if (quad) return d < D ? *reinterpret_cast<const float4*>(p + d) : make_float4(rest, rest, rest, rest);
  return make_float4(d < D ? p[d] : rest, d + 1 < D ? p[d + 1] : rest, d + 2 < D ? p[d + 2] : rest, d + 3 < D ? p[d + 3] : rest);
}

// A warp per value head of a chunk; a lane has NG groups of four channels.  The keys so far, decayed up to the current
// token, stand in registers: every pair of tokens costs a lane one multiplication and two multiply-adds a channel.
template <int NG>
__global__ void __launch_bounds__(kGramWarps * 32) channel_gram_kernel(const DeltaRule a) {
  US_PDL_PROLOGUE();
  __shared__ float low[kGramWarps][kChunk][kChunk + 1], step[kGramWarps][kChunk];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int s, start, n, chunk = blockIdx.x;
  const int h = blockIdx.y * kGramWarps + warp;
  if (!find_chunk(a, s, start, n, chunk) || h >= a.H) return;
  const long long row = start + (long long)chunk * kChunk;
  const int rows = min(kChunk, n - chunk * kChunk), hk = h / (a.H / a.Hk);
  const bool quad = (a.D & 3) == 0 && (a.V & 3) == 0;
  float* out = a.coef + ((first_chunk(start, s) + chunk) * a.H + h) * kCoef;
  if (lane < kChunk) step[warp][lane] = lane < rows ? a.beta[(row + lane) * a.H + h] : 0.f;
  __syncwarp();
  float4 c[kChunk][NG];
#pragma unroll
  for (int t = 0; t < kChunk; ++t) {
    float4 k[NG], q[NG];
    float sum[32];                                   // k_t . (R k_i), then q_t . (R k_i)
#pragma unroll
    for (int e = 0; e < 32; ++e) sum[e] = 0.f;
#pragma unroll
    for (int j = 0; j < NG; ++j) {
      const int d = j * 128 + lane * 4;
      const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
      float4 g = make_float4(1.f, 1.f, 1.f, 1.f);
      k[j] = q[j] = zero;
      if (t < rows) {
        k[j] = load_four(a.k + ((row + t) * a.Hk + hk) * a.D, d, a.D, quad, 0.f);
        q[j] = load_four(a.q + ((row + t) * a.Hk + hk) * a.D, d, a.D, quad, 0.f);
        g = load_four(a.g + ((row + t) * a.H + h) * a.D, d, a.D, quad, 1.f);
      }
#pragma unroll
      for (int i = 0; i < t; ++i) {
        float4& x = c[i][j];
        x = make_float4(x.x * g.x, x.y * g.y, x.z * g.z, x.w * g.w);
        sum[i] = fmaf(x.x, k[j].x, fmaf(x.y, k[j].y, fmaf(x.z, k[j].z, fmaf(x.w, k[j].w, sum[i]))));
        sum[16 + i] = fmaf(x.x, q[j].x, fmaf(x.y, q[j].y, fmaf(x.z, q[j].z, fmaf(x.w, q[j].w, sum[16 + i]))));
      }
      c[t][j] = k[j];
      sum[16 + t] = fmaf(k[j].x, q[j].x, fmaf(k[j].y, q[j].y, fmaf(k[j].z, q[j].z, fmaf(k[j].w, q[j].w, sum[16 + t]))));
    }
    // 32 sums over 32 lanes: lane e ends up with the e-th
#pragma unroll
    for (int w = 16; w >= 1; w >>= 1) {
      const bool up = lane & w;
#pragma unroll
      for (int e = 0; e < w; ++e) {
        const float keep = up ? sum[e + w] : sum[e], give = up ? sum[e] : sum[e + w];
        sum[e] = keep + __shfl_xor_sync(0xffffffffu, give, w);
      }
    }
    if (lane < kChunk) low[warp][t][lane] = step[warp][t] * sum[0];
    else out[kW + t * kChunk + lane - kChunk] = sum[0];
  }
  __syncwarp();
  solve_columns(low[warp], step[warp], out, lane);
}

template <int BYTES>
__device__ __forceinline__ void cp_async(float* dst, const float* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  if (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}

// x = hi + lo, hi rounded to TF32 (the product takes the upper 19 bits of lo).
struct Split {
  uint32_t hi, lo;
  __device__ __forceinline__ Split() {}
  __device__ __forceinline__ explicit Split(float x) {
    hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
    lo = __float_as_uint(x - __uint_as_float(hi));
  }
};

__device__ __forceinline__ void mma_tf32(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_tf32_first(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                               uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

// An accumulator tile as the A operand of the next product: its columns 2 i and 2 i + 1 become k = i and i + 4.
struct Tile {
  Split s[4];
  __device__ __forceinline__ Tile() {}
  __device__ __forceinline__ explicit Tile(const float (&c)[4]) {
#pragma unroll
    for (int e = 0; e < 4; ++e) s[e] = Split(c[e]);
  }
};

// c = a b (first) or c += a b, all of them split: the products with low parts, the product of the high parts.  The
// units add towards zero, so a sum takes all its low products before the first high one.
__device__ __forceinline__ void mma_low(bool first, float (&c)[4], const Tile& a, const Split& b0, const Split& b1) {
  if (first) mma_tf32_first(c, a.s[0].lo, a.s[2].lo, a.s[1].lo, a.s[3].lo, b0.hi, b1.hi);
  else mma_tf32(c, a.s[0].lo, a.s[2].lo, a.s[1].lo, a.s[3].lo, b0.hi, b1.hi);
  mma_tf32(c, a.s[0].hi, a.s[2].hi, a.s[1].hi, a.s[3].hi, b0.lo, b1.lo);
}
__device__ __forceinline__ void mma_high(float (&c)[4], const Tile& a, const Split& b0, const Split& b1) {
  mma_tf32(c, a.s[0].hi, a.s[2].hi, a.s[1].hi, a.s[3].hi, b0.hi, b1.hi);
}

// A chunk in shared memory: k of its tokens, q, with a decay per channel g (then the keys times R_t16), 32 columns of
// v, the coefficients, P_16 per channel.  Rows of k, q, g and v stand 8 banks apart and rows of M and W 4 x 5: every
// load below is then free of conflicts.
template <int DP, bool CHANNEL>
struct Stage {
  static constexpr int kD = DP + 8, kVp = kCols + 8, kMp = kChunk + 4;
  static constexpr int kQ = kChunk * kD, kG = 2 * kChunk * kD, kV = (CHANNEL ? 3 : 2) * kChunk * kD;
  static constexpr int kMat = kV + kChunk * kVp, kVec = kMat + 2 * kChunk * kMp, kAll = kVec + 2 * kChunk;
  static constexpr int kFloats = kAll + (CHANNEL ? DP : 0);
};

// 4093 rows of 16 key and 32 value heads of 128 x 128, one sequence, with the coefficients: a decay per head 791 us four
// tokens at a time, 457 here; a decay per channel 1513 us token by token, 582 here (two sequences of 4050: 1889,
// 881).  64 sequences of five rows: 208 and 199 us before, 165 and 192 here.  The tensor pipe is busy for some 45 % of
// it; the rest are the splits (three instructions a value) and the waits of a chunk's chain, one warp to a scheduler:
// four warps to a tile's channels, each with the whole solve, took longer.
template <int DP, bool CHANNEL>
__global__ void __launch_bounds__(kThreads, DP > 128 ? 1 : 2) chunk_delta_kernel(const DeltaRule a) {
  US_PDL_PROLOGUE();
  using St = Stage<DP, CHANNEL>;
  constexpr int kOwn = DP / kSplit, NJ = kOwn / 16;   // channels of a warp, in pairs of eight-wide tiles
  extern __shared__ __align__(16) float sm[];
  __shared__ __align__(16) float4 parts[2][kTiles][kSplit][4][32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h = blockIdx.y, s = blockIdx.z, hk = h / (a.H / a.Hk), col0 = blockIdx.x * kCols;
  const int start = a.cu[s], T = a.cu[s + 1] - start, slot = a.slots[s];
  if (T <= 0) return;
  if (slot < 0) {                                     // padding: defined rows, no state
    for (int e = tid; e < T * kCols; e += kThreads) {
      const int t = e / kCols, c = col0 + e - t * kCols;
      if (c < a.V) a.out[((long long)(start + t) * a.H + h) * a.V + c] = 0.f;
    }
    return;
  }
  const int chunks = (T + kChunk - 1) / kChunk;
  if (a.D < DP || col0 + kCols > a.V || (T % kChunk) != 0) {      // places that no copy fills: zero
    for (int e = tid; e < kBufs * St::kFloats; e += kThreads) sm[e] = 0.f;
    __syncthreads();
  }
  const bool quad = (a.V & 3) == 0 && (a.D & 3) == 0;
  const long long kstep = (long long)a.Hk * a.D, vstep = (long long)a.H * a.V, gstep = (long long)a.H * a.D;
  const float* kg = a.k + ((long long)start * a.Hk + hk) * a.D;
  const float* qg = a.q + ((long long)start * a.Hk + hk) * a.D;
  const float* gg = a.g + ((long long)start * a.H + h) * a.D;               // per channel
  const float* vg = a.v + ((long long)start * a.H + h) * a.V + col0;
  const float* cg = a.coef + (first_chunk(start, s) * a.H + h) * kCoef;
  auto fetch = [&](int chunk) {                       // (an empty group past the end)
    if (chunk < chunks) {
      float* dst = sm + (chunk % kBufs) * St::kFloats;
      const int t0 = chunk * kChunk, n = min(kChunk, T - t0);
      if (quad) {
        for (int t = warp; t < n; t += kThreads / 32)
#pragma unroll
          for (int d = lane * 4; d < DP; d += 128)
            if (d < a.D) {
              cp_async<16>(dst + t * St::kD + d, kg + (t0 + t) * kstep + d);
              cp_async<16>(dst + St::kQ + t * St::kD + d, qg + (t0 + t) * kstep + d);
              if (CHANNEL) cp_async<16>(dst + St::kG + t * St::kD + d, gg + (t0 + t) * gstep + d);
            }
        const int c = (lane & 7) * 4;
        for (int t = tid >> 3; t < n; t += kThreads / 8)
          if (col0 + c < a.V) cp_async<16>(dst + St::kV + t * St::kVp + c, vg + (t0 + t) * vstep + c);
      } else {
        for (int t = warp; t < n; t += kThreads / 32) {
          for (int d = lane; d < a.D; d += 32) {
            cp_async<4>(dst + t * St::kD + d, kg + (t0 + t) * kstep + d);
            cp_async<4>(dst + St::kQ + t * St::kD + d, qg + (t0 + t) * kstep + d);
            if (CHANNEL) cp_async<4>(dst + St::kG + t * St::kD + d, gg + (t0 + t) * gstep + d);
          }
          if (col0 + lane < a.V) cp_async<4>(dst + St::kV + t * St::kVp + lane, vg + (t0 + t) * vstep + lane);
        }
      }
      const float* src = cg + (long long)chunk * a.H * kCoef;
#pragma unroll
      for (int e = tid * 4; e < 2 * kChunk * kChunk; e += kThreads * 4)      // both matrices, row by row
        cp_async<16>(dst + St::kMat + e / kChunk * St::kMp + e % kChunk, src + e);
      if (!CHANNEL && tid < 2 * kChunk / 4) cp_async<16>(dst + St::kVec + tid * 4, src + kP + tid * 4);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // keys and queries times P_t, keys times R_t16 in the decays' place, P_16; a thread per channel
  auto decayed = [&](int chunk) {
    float* b = sm + (chunk % kBufs) * St::kFloats;
    const int n = min(kChunk, T - chunk * kChunk);
    for (int d = tid; d < DP; d += kThreads) {
      float g[kChunk], k[kChunk], p = 1.f, r = 1.f;
#pragma unroll
      for (int t = 0; t < kChunk; ++t) {
        const bool in = t < n && d < a.D;
        g[t] = in ? b[St::kG + t * St::kD + d] : 1.f;
        k[t] = in ? b[t * St::kD + d] : 0.f;
        p *= g[t];
        b[t * St::kD + d] = k[t] * p;
        b[St::kQ + t * St::kD + d] *= p;
      }
      b[St::kAll + d] = p;
#pragma unroll
      for (int t = kChunk - 1; t >= 0; --t) {
        b[St::kG + t * St::kD + d] = k[t] * r;
        r *= g[t];
      }
    }
  };
#pragma unroll 1
  for (int f = 0; f < kBufs - 1; ++f) fetch(f);
  const int tile = warp / kSplit, half = warp % kSplit, r = lane >> 2, i = lane & 3;
  // A tile's columns 2 i and 2 i + 1 are tokens i and 4 + (i ^ 2) of eight: loads of rows by column number and by
  // column pair then both meet every bank once.
  const int t0 = i, t1 = 4 + (i ^ 2), tr = (r & 1) ? 4 + ((r >> 1) ^ 2) : r >> 1;
  const int col = col0 + tile * 16 + r, dbase = half * kOwn;
  float* Sg = a.state + ((long long)slot * a.H + h) * a.D * a.V;
  const bool fresh = a.pos && a.pos[start] == 0;
  // S^T: tile (j, e) has columns n = channel 16 j + 2 n + e of the warp's
  float S[NJ][2][4];
#pragma unroll
  for (int j = 0; j < NJ; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int d = dbase + 16 * j + 4 * i + 2 * (c & 1) + e, v = col + (c >> 1) * 8;
        S[j][e][c] = !fresh && d < a.D && v < a.V ? Sg[(long long)d * a.V + v] : 0.f;
      }
  float* op = a.out + ((long long)start * a.H + h) * a.V + col;
  const long long ostep = (long long)a.H * a.V;
  if (CHANNEL) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kBufs - 2) : "memory");
    __syncthreads();
    decayed(0);
  }
  for (int ch = 0; ch < chunks; ++ch) {
    // this chunk's vectors are there (decayed ones: and the next chunk's), the one before is consumed
    asm volatile("cp.async.wait_group %0;" ::"n"(CHANNEL ? 0 : kBufs - 2) : "memory");
    __syncthreads();
    fetch(ch + kBufs - 1);
    if (CHANNEL && ch + 1 < chunks) decayed(ch + 1);
    const float* base = sm + (ch % kBufs) * St::kFloats;
    const float* M = base + St::kMat;
    const float* vec = base + St::kVec;
    // What keys (tiles 0, 1) and queries (2, 3) see of S0, over this warp's channels.  As the units add towards
    // zero, no sum of theirs is longer than two steps of channels; longer ones and the state's are rounded.
    float x[4][4];
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const Tile s0(S[j][0]), s1(S[j][1]);
      float4 f[4];
#pragma unroll
      for (int n = 0; n < 4; ++n)
        f[n] = *reinterpret_cast<const float4*>(base + (n >> 1) * St::kQ + ((n & 1) * 8 + tr) * St::kD + dbase + 16 * j + 4 * i);
      float y[4][4];
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const Split bx(f[n].x), by(f[n].y), bz(f[n].z), bw(f[n].w);
        mma_low(true, y[n], s0, bx, bz);
        mma_low(false, y[n], s1, by, bw);
        mma_high(y[n], s0, bx, bz);
        mma_high(y[n], s1, by, bw);
      }
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int c = 0; c < 4; ++c) x[n][c] = j ? x[n][c] + y[n][c] : y[n][c];
    }
    float4(*mine)[32] = parts[ch & 1][tile][half];
#pragma unroll
    for (int n = 0; n < 4; ++n) mine[n][lane] = make_float4(x[n][0], x[n][1], x[n][2], x[n][3]);
    asm volatile("bar.sync %0, %1;" ::"r"(1 + tile), "n"(32 * kSplit) : "memory");
#pragma unroll
    for (int o = 1; o < kSplit; ++o) {
      const float4(*other)[32] = parts[ch & 1][tile][(half + o) % kSplit];
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        if (n >= 2 && n % kSplit != half) continue;   // queries of another warp's tokens
        const float4 y = other[n][lane];
        x[n][0] += y.x;
        x[n][1] += y.y;
        x[n][2] += y.z;
        x[n][3] += y.w;
      }
    }
    // U = M (V - P X)
    Tile res[2];
    float p[2][2];
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      p[n][0] = CHANNEL ? 1.f : vec[n * 8 + t0];
      p[n][1] = CHANNEL ? 1.f : vec[n * 8 + t1];
      float w[4];
#pragma unroll
      for (int c = 0; c < 4; ++c)
        w[c] = fmaf(-p[n][c & 1], x[n][c],
                    base[St::kV + (n * 8 + ((c & 1) ? t1 : t0)) * St::kVp + tile * 16 + r + (c >> 1) * 8]);
      res[n] = Tile(w);
    }
    float u[2][4], u1[4];
    const float* at = M + tr * St::kMp;
    const Split m0(at[t0]), m1(at[t1]), m2(at[8 * St::kMp + t0]), m3(at[8 * St::kMp + t1]);
    const Split m4(at[8 * St::kMp + 8 + t0]), m5(at[8 * St::kMp + 8 + t1]);
    mma_low(true, u[0], res[0], m0, m1);
    mma_low(true, u[1], res[0], m2, m3);
    mma_low(true, u1, res[1], m4, m5);
    mma_high(u[0], res[0], m0, m1);
    mma_high(u[1], res[0], m2, m3);
    mma_high(u1, res[1], m4, m5);
#pragma unroll
    for (int c = 0; c < 4; ++c) u[1][c] += u1[c];
    const Tile ut[2] = {Tile(u[0]), Tile(u[1])};
    // S' = P_16 S0 + (R K)^T U
    Tile wr[2];
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      if (CHANNEL) {
        wr[n] = ut[n];
      } else {
        const float r0 = vec[kChunk + n * 8 + t0], r1 = vec[kChunk + n * 8 + t1];
        const float w[4] = {u[n][0] * r0, u[n][1] * r1, u[n][2] * r0, u[n][3] * r1};
        wr[n] = Tile(w);
      }
    }
    const float* kr = base + (CHANNEL ? St::kG : 0);
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      float y[2][4];
      Split b[2][2][2];
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const float2 f0 = *reinterpret_cast<const float2*>(kr + (n * 8 + t0) * St::kD + dbase + 16 * j + 2 * r);
        const float2 f1 = *reinterpret_cast<const float2*>(kr + (n * 8 + t1) * St::kD + dbase + 16 * j + 2 * r);
        b[n][0][0] = Split(f0.x);
        b[n][0][1] = Split(f1.x);
        b[n][1][0] = Split(f0.y);
        b[n][1][1] = Split(f1.y);
#pragma unroll
        for (int e = 0; e < 2; ++e) mma_low(n == 0, y[e], wr[n], b[n][e][0], b[n][e][1]);
      }
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) mma_high(y[e], wr[n], b[n][e][0], b[n][e][1]);
      float4 all;
      if (CHANNEL) all = *reinterpret_cast<const float4*>(base + St::kAll + dbase + 16 * j + 4 * i);
      else all.x = all.y = all.z = all.w = vec[kChunk - 1];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        S[j][0][c] = fmaf(S[j][0][c], (c & 1) ? all.z : all.x, y[0][c]);
        S[j][1][c] = fmaf(S[j][1][c], (c & 1) ? all.w : all.y, y[1][c]);
      }
    }
    // O = P Q S0 + W U: a tile of eight tokens per warp
    const float* W = M + kChunk * St::kMp;
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      if (n % kSplit != half) continue;
      float o[4];
      Split b[2][2];
#pragma unroll
      for (int m = 0; m <= n; ++m) {
        const float* wt = W + (n * 8 + tr) * St::kMp + m * 8;
        b[m][0] = Split(wt[t0]);
        b[m][1] = Split(wt[t1]);
        mma_low(m == 0, o, ut[m], b[m][0], b[m][1]);
      }
#pragma unroll
      for (int m = 0; m <= n; ++m) mma_high(o, ut[m], b[m][0], b[m][1]);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int t = ch * kChunk + n * 8 + ((c & 1) ? t1 : t0);
        if (t < T && col + (c >> 1) * 8 < a.V) op[t * ostep + (c >> 1) * 8] = fmaf(x[2 + n][c], p[n][c & 1], o[c]);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < NJ; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int d = dbase + 16 * j + 4 * i + 2 * (c & 1) + e, v = col + (c >> 1) * 8;
        if (d < a.D && v < a.V) Sg[(long long)d * a.V + v] = S[j][e][c];
      }
}

template <int DP, bool CHANNEL>
int launch(const DeltaRule& a, cudaStream_t stream) {
  constexpr int need = kBufs * Stage<DP, CHANNEL>::kFloats * sizeof(float);
  constexpr int alone = need > 110 * 1024 ? need : 110 * 1024;      // shared memory that one CTA per SM has
  static bool configured = false;
  static int sms = 0;
  if (!configured) {
    int dev = 0;
    US_CUDA_CHECK(cudaGetDevice(&dev));
    US_CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    US_CUDA_CHECK(cudaFuncSetAttribute(chunk_delta_kernel<DP, CHANNEL>, cudaFuncAttributeMaxDynamicSharedMemorySize, alone));
    configured = true;
  }
  // CTAs that are launched while the kernel before still runs would be packed two to an SM where it
  // leaves room: with fewer CTAs than SMs each asks for more shared memory than half an SM has
  const dim3 grid(us::ceil_div(a.V, kCols), a.H, a.B);
  const size_t smem = (long long)grid.x * grid.y * grid.z <= sms ? alone : need;
  US_CUDA_CHECK(us::launch_pdl(chunk_delta_kernel<DP, CHANNEL>, grid, dim3(kThreads), smem, stream, a));
  return US_OK;
}

int run(const DeltaRule& a, int rows, bool channel, cudaStream_t stream) {
  US_REQUIRE(a.q && a.k && a.v && a.g && a.beta && a.coef && a.state && a.out && a.cu && a.slots);
  US_REQUIRE(a.B >= 1 && a.B <= 65535 && rows >= 0 && a.H >= 1 && a.Hk >= 1 && a.H % a.Hk == 0 && a.H <= 65535);
  US_REQUIRE(a.D >= 1 && a.V >= 1 && ((uintptr_t)a.coef % 16) == 0);
  US_REQUIRE((a.D & 3) || (a.V & 3) || (((uintptr_t)a.q | (uintptr_t)a.k | (uintptr_t)a.v | (channel ? (uintptr_t)a.g : 0)) % 16) == 0);
  if (a.D > kMaxDim) return US_ERR_UNSUPPORTED;
  if (rows == 0) return US_OK;
  const dim3 grams(rows / kChunk + a.B, us::ceil_div(channel ? a.H : a.Hk, kGramWarps)), threads(kGramWarps * 32);
  auto gram = !channel ? head_gram_kernel : a.D <= 128 ? channel_gram_kernel<1> : channel_gram_kernel<2>;
  US_CUDA_CHECK(us::launch_pdl(gram, grams, threads, 0, stream, a));
  if (a.D <= 64) return channel ? launch<64, true>(a, stream) : launch<64, false>(a, stream);
  if (a.D <= 128) return channel ? launch<128, true>(a, stream) : launch<128, false>(a, stream);
  return channel ? launch<256, true>(a, stream) : launch<256, false>(a, stream);
}

}  // namespace

US_API long long us_delta_coef_floats(int rows, int B, int H) { return ((long long)rows / kChunk + B + 1) * H * kCoef; }

// q and k heads serve H / Hk value heads each; all vectors dense FP32; coef: scratch of
// us_delta_coef_floats floats; pos null: every sequence goes on from its slot's state.
US_API int us_head_delta_rule(const float* q, const float* k, const float* v, const float* g,
                              const float* beta, float* coef, float* state, float* out, const int* cu,
                              const int* slots, const int* pos, int B, int rows, int H, int Hk, int D, int V,
                              void* stream) {
  return run(DeltaRule{q, k, v, g, beta, coef, state, out, cu, slots, pos, B, H, Hk, D, V}, rows, false, (cudaStream_t)stream);
}

// The same with g [rows, H, D].
US_API int us_channel_delta_rule(const float* q, const float* k, const float* v, const float* g,
                                 const float* beta, float* coef, float* state, float* out, const int* cu,
                                 const int* slots, const int* pos, int B, int rows, int H, int Hk, int D, int V,
                                 void* stream) {
  return run(DeltaRule{q, k, v, g, beta, coef, state, out, cu, slots, pos, B, H, Hk, D, V}, rows, true, (cudaStream_t)stream);
}
