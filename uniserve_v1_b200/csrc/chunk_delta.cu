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
// The chain from chunk to chunk is three small products.  They run on the tensor cores with FP32 operands in three
// bf16 parts, which hold all 24 bits, and the six products of parts that reach them (what is left out is 2^-25 of a
// product and less).  The units round sums towards zero.  So products of leading parts are summed over sixteen
// channels or tokens at a time, from zero, and added on the FP32 units; the leading part of every operand but the state
// and U has only six bits, which leaves such a sum room for nearly all of its bits; the smaller products have a sum of
// their own.  Token by token, or four tokens at a time on the FP32 units, a chunk took sixteen or four rounds of
// shuffles and dependent sums.  mma.sync and not tcgen05: a chunk's operands come from registers (the state's
// accumulators are the next product's A operand as they stand), and a round through tensor memory costs more than
// these products do.
//
// A CTA owns 32 value columns of one head of one sequence.  Four warps carry the chain: two tiles of sixteen columns,
// each two warps that share the channels.  Such a warp holds S^T [16 columns, D / 2 channels] as accumulators.  Partial
// K S0 and Q S0 meet in shared memory; both warps of a tile solve U.  Four more warps do what is not on the chain: they
// fetch the next chunk's vectors, multiply them with their decays where those are per channel, and lay their parts out
// in shared memory, two chunks at most, and they form a chunk's outputs while the next one is under way.  A sequence
// whose first packed row stands at position 0 starts from a zero state whatever its slot holds; a negative slot marks
// padding.
//
// Values that are not finite stay where the recurrence has them.  M and W are lower triangular, and as matrix
// operands their zeros would carry a token's infinity or NaN to the tokens before it; a tile whose U is not finite
// everywhere takes its sums over the tokens up to each one instead.
#include "include/us_common.cuh"
#include "include/us_f32x2.cuh"
#include "include/us_mma.cuh"

namespace {

using namespace us::f32x2;

constexpr int kChunk = 16;        // tokens whose products share a state
constexpr int kCols = 32;         // value columns per CTA
constexpr int kSplit = 2;         // warps that share a tile's channels
constexpr int kTiles = kCols / 16;
constexpr int kCompute = 32 * kSplit * kTiles, kFeed = 128, kThreads = kCompute + kFeed;
constexpr int kMaxDim = 256;

// Coefficients of a chunk and head: M [t][i] and W [t][i] below their diagonals, as three bf16 parts each | beta_t and
// W_tt, the diagonals | with a decay per head P_t | R_t16
constexpr int kMat = 3 * kChunk * kChunk / 2, kDiag = 2 * kMat, kP = kDiag + 2 * kChunk, kCoef = kP + 2 * kChunk;

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

// x to six bits; what remains of it is the sum of two bf16
__device__ __forceinline__ float leading(float x) {
  return __uint_as_float((__float_as_uint(x) + 0x20000u) & 0xfffc0000u);
}
// (x, y) = sum of three bf16 pairs, the first of six bits each
__device__ __forceinline__ void split(float x, float y, uint32_t (&o)[3]) {
  const float a = leading(x), b = leading(y);
  o[0] = us::pack_bf(a, b);
  x -= a;
  y -= b;
#pragma unroll
  for (int i = 1; i < 3; ++i) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(x, y);
    o[i] = *reinterpret_cast<const uint32_t*>(&p);
    x -= us::bf2f(p.x);
    y -= us::bf2f(p.y);
  }
}

// Eight neighbours of row t of matrix 0 (M) or 1 (W), what stands below the diagonal.
__device__ __forceinline__ void put_coefs(float* coef, int matrix, int t, int i0, const float (&x)[8]) {
  uint32_t o[4][3];
#pragma unroll
  for (int e = 0; e < 4; ++e)
    split(i0 + 2 * e < t ? x[2 * e] : 0.f, i0 + 2 * e + 1 < t ? x[2 * e + 1] : 0.f, o[e]);
#pragma unroll
  for (int p = 0; p < 3; ++p)
    *reinterpret_cast<uint4*>(coef + matrix * kMat + (p * kChunk * kChunk + t * kChunk + i0) / 2) =
        make_uint4(o[0][p], o[1][p], o[2][p], o[3][p]);
}

// M from L (strictly lower) and beta, by forward substitution: a lane per column, then a lane per half a row.
__device__ __forceinline__ void solve(float (*low)[kChunk + 1], const float* beta, float* out, int lane) {
  float m[kChunk];
  if (lane < kChunk) {
#pragma unroll
    for (int x = 0; x < kChunk; ++x) {
      float sum = x == lane ? beta[x] : 0.f;
#pragma unroll
      for (int y = 0; y < x; ++y) sum = fmaf(-low[x][y], m[y], sum);
      m[x] = sum;
    }
  }
  __syncwarp();
  if (lane < kChunk) {
#pragma unroll
    for (int x = 0; x < kChunk; ++x) low[x][lane] = m[x];
    out[kDiag + lane] = beta[lane];
  }
  __syncwarp();
  const int t = lane >> 1, i0 = (lane & 1) * 8;
  float row[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) row[e] = low[t][i0 + e];
  put_coefs(out, 0, t, i0, row);
}

__device__ __forceinline__ float dot4(const float4& x, const float4& y, float sum) {
  return fmaf(x.x, y.x, fmaf(x.y, y.y, fmaf(x.z, y.z, fmaf(x.w, y.w, sum))));
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
    float k32[8], q32[8];                            // chains of eight products, then of 32: short ones round less
#pragma unroll
    for (int e = 0; e < 8; ++e) k32[e] = q32[e] = 0.f;
#pragma unroll
    for (int d = 0; d < 32; d += 8) {
      const float4 kt = *reinterpret_cast<const float4*>(kr + t * kGramPitch + d);
      const float4 qt = *reinterpret_cast<const float4*>(qr + t * kGramPitch + d);
      const float4 kt4 = *reinterpret_cast<const float4*>(kr + t * kGramPitch + d + 4);
      const float4 qt4 = *reinterpret_cast<const float4*>(qr + t * kGramPitch + d + 4);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float4 ki = *reinterpret_cast<const float4*>(kr + (i0 + e) * kGramPitch + d);
        const float4 ki4 = *reinterpret_cast<const float4*>(kr + (i0 + e) * kGramPitch + d + 4);
        k32[e] += dot4(kt, ki, dot4(kt4, ki4, 0.f));
        q32[e] += dot4(qt, ki, dot4(qt4, ki4, 0.f));
      }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      kk[e] += k32[e];
      qk[e] += q32[e];
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
    double r = 1.;                                   // g_(i+1) .. g_t, from i = t down to this lane's tokens
    for (int i = t - 1; i >= i0 + 8; --i) r *= g[i + 1];
    float w[8];
#pragma unroll
    for (int e = 7; e >= 0; --e) {
      const int i = i0 + e;
      if (i < t) r *= g[i + 1];
      low[warp][t][i] = i < t ? beta_t * (float)r * kk[e] : 0.f;
      w[e] = (float)r * qk[e];
      if (i == t) out[kDiag + kChunk + t] = qk[e];
    }
    put_coefs(out, 1, t, i0, w);
    if (lane < kChunk) {                             // (rounded once: what a head forgets is common to all its state)
      double p = 1., tail = 1.;
      for (int x = 0; x <= lane; ++x) p *= g[x];
      for (int x = lane + 1; x < kChunk; ++x) tail *= g[x];
      out[kP + lane] = (float)p;
      out[kP + kChunk + lane] = (float)tail;
    }
    __syncwarp();
    solve(low[warp], decay[warp][1], out, lane);
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
  __shared__ float low[kGramWarps][kChunk][kChunk + 1], read[kGramWarps][kChunk][kChunk + 1], step[kGramWarps][kChunk];
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
    else read[warp][t][lane - kChunk] = sum[0];
    if (lane == kChunk + t) out[kDiag + lane] = sum[0];
  }
  __syncwarp();
  const int t = lane >> 1, i0 = (lane & 1) * 8;
  float w[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) w[e] = read[warp][t][i0 + e];
  put_coefs(out, 1, t, i0, w);
  solve(low[warp], step[warp], out, lane);
}

// An accumulator tile [16 x 8]: a lane's rows are r and r + 8, its columns 2 i and 2 i + 1.
using Acc = f2[2];

// An A operand [16 x 16] in three parts, from two accumulator tiles that stand side by side.
struct Parts {
  uint32_t p[3][4];
  __device__ __forceinline__ Parts(const Acc& a, const Acc& b) {
    uint32_t o[3];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const f2 x = (e < 2 ? a : b)[e & 1];
      us::split3(lo2(x), hi2(x), o);
#pragma unroll
      for (int n = 0; n < 3; ++n) p[n][e] = o[n];
    }
  }
};

__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_first(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// Four B operands' tiles of one part, two to a load: tile n is b[n / 2][n % 2 * 2 ..]
using Tiles = uint32_t[2][4];
__device__ __forceinline__ void mma4(bool first, float (&c)[4][4], const uint32_t (&a)[4], const Tiles& b) {
#pragma unroll
  for (int n = 0; n < 4; ++n) {
    if (first) mma_first(c[n], a, b[n >> 1][(n & 1) * 2], b[n >> 1][(n & 1) * 2 + 1]);
    else mma(c[n], a, b[n >> 1][(n & 1) * 2], b[n >> 1][(n & 1) * 2 + 1]);
  }
}
// Products of `a` and four tiles, whose part p `load(b, p)` brings: high = those of the leading parts, low += the five
// smaller ones (first: low = them).  Four sums side by side cover an instruction's latency.
template <typename Load>
__device__ __forceinline__ void products(bool first, float (&high)[4][4], float (&low)[4][4], const Parts& a, Load load) {
  Tiles b;
  load(b, 2);
  mma4(first, low, a.p[0], b);
  load(b, 1);
  mma4(false, low, a.p[1], b);
  mma4(false, low, a.p[0], b);
  load(b, 0);
  mma4(false, low, a.p[2], b);
  mma4(false, low, a.p[1], b);
  mma4(true, high, a.p[0], b);
}

// A chunk in shared memory, in bytes: arrays [part][token][channel] bf16 of k, of q and, with a decay per channel, of
// k R_t16 (k and q then times P_t), rows 16 bytes past a multiple of 128; 32 columns of v (rows 4 banks apart); M and W
// [part][t][i] (rows of 48 bytes); beta_t, W_tt, P_t and R_t16, or P_16 of every channel in place of the last two; the
// last four tokens' k (k R_t16) whole, of sixteen channels those of a lane side by side.  Every load of them is free of conflicts.
constexpr int kLast = 4;
template <int DP, bool CHANNEL>
struct Stage {
  static constexpr int kRow = (DP + 8) * 2, kPart = kChunk * kRow, kArray = 3 * kPart;
  static constexpr int kQ = kArray, kKr = (CHANNEL ? 2 : 0) * kArray, kV = (CHANNEL ? 3 : 2) * kArray;
  static constexpr int kVp = kCols + 4, kCoefs = kV + kChunk * kVp * 4, kCoefRow = 48, kCoefPart = kChunk * kCoefRow;
  static constexpr int kVec = kCoefs + 6 * kCoefPart, kAll = kVec + 2 * kChunk * 4;
  static constexpr int kTail = kAll + (CHANNEL ? DP : 2 * kChunk) * 4, kBytes = kTail + kLast * DP * 4;
};

// Named barriers.  Each has a second one for chunks of the other parity: a warp that arrives without waiting may be a
// chunk ahead of those that wait, never two, since the next chunk but one is only laid out once this one is done with.
enum Barrier : int { kTileBar = 1, kFullBar = 3, kEmptyBar = 5, kWritesBar = 7 };
__device__ __forceinline__ void bar_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// What the warps of a chunk hand on: [chunk parity][tile][half of the channels][K S0, Q S0 of eight tokens][lane],
// accumulator tiles over that half.  In place of the first two of the other half, once they are read, U.
using Exchange = float4[2][kTiles][kSplit][4][32];
// entry (column, token) of two tiles [16 columns x 8 tokens] that stand side by side
__device__ __forceinline__ float entry(const float4 (*x)[32], int col, int t) {
  return reinterpret_cast<const float*>(&x[t >> 3][(col & 7) * 4 + ((t & 7) >> 1)])[(col >> 3) * 2 + (t & 1)];
}
// an FP32 value from its three parts
__device__ __forceinline__ float whole(const unsigned char* at, int part) {
  float sum = 0.f;
#pragma unroll
  for (int q = 2; q >= 0; --q) sum += us::bf2f(*reinterpret_cast<const __nv_bfloat16*>(at + q * part));
  return sum;
}
// row t of M (0) or W (1) times a column, over the tokens up to t
template <typename St>
__device__ __forceinline__ float row_sum(const unsigned char* base, int matrix, int t, const float4 (*x)[32], int col) {
  const unsigned char* row = base + St::kCoefs + matrix * 3 * St::kCoefPart + t * St::kCoefRow;
  float sum = 0.f;
#pragma unroll 1
  for (int y = 0; y < t; ++y) sum = fmaf(whole(row + y * 2, St::kCoefPart), entry(x, col, y), sum);
  return fmaf(reinterpret_cast<const float*>(base + St::kVec)[matrix * kChunk + t], entry(x, col, t), sum);
}
__device__ __forceinline__ bool all_finite(const Acc& a, const Acc& b) {
  const f2 zero = pack2(0.f, 0.f);
  const f2 x = fma2(b[0], zero, mul2(a[0], zero)), y = fma2(b[1], zero, mul2(a[1], zero));
  const f2 sum = add2(x, y);
  return !__any_sync(0xffffffffu, lo2(sum) + hi2(sum) != 0.f);
}

// The warps that feed: a chunk's vectors are on their way to registers while the one before is multiplied.
template <int DP, bool CHANNEL>
struct Feeder {
  using St = Stage<DP, CHANNEL>;
  static constexpr int kMine = kChunk * DP / 4 / kFeed;     // tokens of four channels
  // With a decay per channel a thread has the same four channels of kMine tokens in turn, and the threads of a warp
  // that share them stand kFours lanes apart; else it has pieces all over the chunk.
  static constexpr int kFours = 32 * kMine / kChunk;
  const DeltaRule& a;
  const float *k, *q, *g, *v, *coef;
  long long kstep, vstep, gstep;
  int tid, T, col0, D;
  bool quad;
  float4 kv[kMine], qv[kMine], gv[CHANNEL ? kMine : 1], vv, cc[2];
  __device__ __forceinline__ Feeder(const DeltaRule& a_, int tid_, int start, int s, int T_, int h, int hk, int col0_)
      : a(a_), tid(tid_), T(T_), col0(col0_), D(a_.D) {
    kstep = (long long)a.Hk * a.D;
    vstep = (long long)a.H * a.V;
    gstep = (long long)a.H * a.D;
    k = a.k + ((long long)start * a.Hk + hk) * a.D;
    q = a.q + ((long long)start * a.Hk + hk) * a.D;
    g = a.g + ((long long)start * a.H + h) * a.D;
    v = a.v + ((long long)start * a.H + h) * a.V;
    coef = a.coef + (first_chunk(start, s) * a.H + h) * kCoef;
    quad = (a.V & 3) == 0 && (a.D & 3) == 0;
  }
  __device__ __forceinline__ int token(int i) const {
    return CHANNEL ? (tid & 31) / kFours * kMine + i : (tid + i * kFeed) / (DP / 4);
  }
  __device__ __forceinline__ int channel(int i) const {
    return 4 * (CHANNEL ? (tid >> 5) * kFours + (tid & (kFours - 1)) : (tid + i * kFeed) % (DP / 4));
  }
  __device__ __forceinline__ void load(int chunk) {
    const int t0 = chunk * kChunk, n = T - t0;
#pragma unroll
    for (int i = 0; i < kMine; ++i) {
      const int t = token(i), d = channel(i);
      kv[i] = qv[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (CHANNEL) gv[i] = make_float4(1.f, 1.f, 1.f, 1.f);
      if (t < n && d < D) {
        kv[i] = load_four(k + (t0 + t) * kstep, d, D, quad, 0.f);
        qv[i] = load_four(q + (t0 + t) * kstep, d, D, quad, 0.f);
        if (CHANNEL) gv[i] = load_four(g + (t0 + t) * gstep, d, D, quad, 1.f);
      }
    }
    const int t = tid >> 3, c = col0 + (tid & 7) * 4;
    vv = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t < n && c < a.V) vv = load_four(v + (t0 + t) * vstep, c, a.V, quad, 0.f);
    const float4* m = reinterpret_cast<const float4*>(coef + (long long)chunk * a.H * kCoef);
    cc[0] = m[tid];
    if (tid < (CHANNEL ? kP : kCoef) / 4 - kFeed) cc[1] = m[tid + kFeed];
  }
  __device__ __forceinline__ static void put(unsigned char* at, const float4& x) {
    uint32_t o[3], u[3];
    split(x.x, x.y, o);
    split(x.z, x.w, u);
#pragma unroll
    for (int p = 0; p < 3; ++p) *reinterpret_cast<uint2*>(at + p * St::kPart) = make_uint2(o[p], u[p]);
  }
  __device__ __forceinline__ void last(unsigned char* b, int i, const float4& x) const {
    const int t = token(i) - (kChunk - kLast), d = channel(i), at = t * DP + d / 16 * 16 + (d & 7) * 2 + (d & 8) / 4;
    *reinterpret_cast<float2*>(b + St::kTail + at * 4) = make_float2(x.x, x.y);
    *reinterpret_cast<float2*>(b + St::kTail + (at + 4) * 4) = make_float2(x.z, x.w);
  }
  __device__ __forceinline__ static float4 mul(const float4& x, const float4& y) {
    return make_float4(x.x * y.x, x.y * y.y, x.z * y.z, x.w * y.w);
  }
  __device__ __forceinline__ void store(unsigned char* b) const {
    const int d0 = channel(0);
    float4 p, r;                                      // decays from the chunk's start, and to its end
    if (CHANNEL) {
      float4 all = make_float4(1.f, 1.f, 1.f, 1.f);   // of this thread's tokens
      p = r = all;
#pragma unroll
      for (int i = 0; i < kMine; ++i) all = mul(all, gv[i]);
      const int mine = (tid & 31) / kFours;
#pragma unroll
      for (int s = 0; s < 32 / kFours; ++s) {
        const int from = s * kFours + (tid & (kFours - 1));
        const float4 x = make_float4(__shfl_sync(0xffffffffu, all.x, from), __shfl_sync(0xffffffffu, all.y, from),
                                     __shfl_sync(0xffffffffu, all.z, from), __shfl_sync(0xffffffffu, all.w, from));
        if (s < mine) p = mul(p, x);
        if (s > mine) r = mul(r, x);
      }
    }
#pragma unroll
    for (int i = 0; i < kMine; ++i) {
      if (CHANNEL) p = mul(p, gv[i]);
      unsigned char* at = b + token(i) * St::kRow + channel(i) * 2;
      put(at, CHANNEL ? mul(kv[i], p) : kv[i]);
      if (!CHANNEL && token(i) >= kChunk - kLast) last(b, i, kv[i]);
      put(at + St::kQ, CHANNEL ? mul(qv[i], p) : qv[i]);
    }
    if (CHANNEL) {
      if ((tid & 31) / kFours == 32 / kFours - 1) *reinterpret_cast<float4*>(b + St::kAll + d0 * 4) = p;
#pragma unroll
      for (int i = kMine - 1; i >= 0; --i) {
        const float4 x = mul(kv[i], r);
        put(b + St::kKr + token(i) * St::kRow + d0 * 2, x);
        if (token(i) >= kChunk - kLast) last(b, i, x);
        r = mul(r, gv[i]);
      }
    }
    *reinterpret_cast<float4*>(b + St::kV + ((tid >> 3) * St::kVp + (tid & 7) * 4) * 4) = vv;
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const int e = tid + n * kFeed;                  // pieces of 16 bytes: two to a row of M and W
      if (e < kDiag / 4) *reinterpret_cast<float4*>(b + St::kCoefs + (e >> 1) * St::kCoefRow + (e & 1) * 16) = cc[n];
      else if (e < (CHANNEL ? kP : kCoef) / 4) *reinterpret_cast<float4*>(b + St::kVec + (e - kDiag / 4) * 16) = cc[n];
    }
  }
  // O = P Q S0 + W U of eight of a chunk's tokens and sixteen columns
  __device__ __forceinline__ void read_out(const unsigned char* b, const Exchange& ex, int chunk, float* out) const {
    const int warp = tid >> 5, lane = tid & 31, tile = warp / kSplit, half = warp % kSplit, r = lane >> 2, i = lane & 3;
    const float4(*parts)[4][32] = ex[chunk & 1][tile];
    const float4(*u)[32] = parts[half ^ 1];
    const float4 seen0 = parts[0][2 + half][lane], seen1 = parts[1][2 + half][lane], u0 = u[0][lane], u1 = u[1][lane];
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(b) + St::kCoefs + 3 * St::kCoefPart +
                        (half * 8 + (lane & 7)) * St::kCoefRow + ((lane >> 3) & 1) * 16;
    uint32_t w01[4], w22[4];
    us::ldsm4(w01, at + (lane >> 4) * St::kCoefPart);                 // two parts
    us::ldsm4(w22, at + 2 * St::kCoefPart);
    const float* vec = reinterpret_cast<const float*>(b + St::kVec) + kChunk + half * 8 + 2 * i;
    const float2 diag = *reinterpret_cast<const float2*>(vec);
    const float2 p = CHANNEL ? make_float2(1.f, 1.f) : *reinterpret_cast<const float2*>(vec + kChunk);
    const Acc ua = {pack2(u0.x, u0.y), pack2(u0.z, u0.w)}, ub = {pack2(u1.x, u1.y), pack2(u1.z, u1.w)};
    float o[4];
    if (__builtin_expect(all_finite(ua, ub), 1)) {
      const Parts up(ua, ub);
      float a1[4], a2[4];
      mma_first(a2, up.p[0], w22[0], w22[1]);
      mma_first(a1, up.p[0], w01[2], w01[3]);
      mma_first(o, up.p[0], w01[0], w01[1]);
      mma(a2, up.p[1], w01[2], w01[3]);
      mma(a1, up.p[1], w01[0], w01[1]);
      mma(a2, up.p[2], w01[0], w01[1]);
      const float4 mine = half ? u1 : u0;
      o[0] = fmaf(diag.x, mine.x, o[0] + (a1[0] + a2[0]));
      o[1] = fmaf(diag.y, mine.y, o[1] + (a1[1] + a2[1]));
      o[2] = fmaf(diag.x, mine.z, o[2] + (a1[2] + a2[2]));
      o[3] = fmaf(diag.y, mine.w, o[3] + (a1[3] + a2[3]));
    } else {
#pragma unroll
      for (int c = 0; c < 4; ++c) o[c] = row_sum<St>(b, 1, half * 8 + 2 * i + (c & 1), u, r + (c >> 1) * 8);
    }
    const float seen[4] = {seen0.x + seen1.x, seen0.y + seen1.y, seen0.z + seen1.z, seen0.w + seen1.w};
    const int col = col0 + tile * 16 + r;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int t = chunk * kChunk + half * 8 + 2 * i + (c & 1), v = col + (c >> 1) * 8;
      if (t < T && v < a.V) out[t * vstep + v] = fmaf(seen[c], (c & 1) ? p.y : p.x, o[c]);
    }
  }
};

// 4093 rows of 16 key and 32 value heads of 128 x 128, one sequence, with the coefficients: a decay per head 790 us four
// tokens at a time, 522 here; a decay per channel 1516 us token by token, 618 here (two sequences of 4050: 1146 -> 930,
// 1887 -> 1122).  Operands in two TF32 parts and three products took 456 and 582, but left results up to 3.1 times as
// far from 64 bits as the FP32 recurrence's; this form's are 0.5 to 1.05 of it (state 1.15 where a token forgets half).
// What bounds it is the chain: 162 tensor instructions of a warp take 1300 of a chunk's 3700 clocks; the rest are the
// splits (eleven instructions a pair of values) and waits, one warp of the chain to a scheduler.
template <int DP, bool CHANNEL, int PER_SM>
__global__ void __launch_bounds__(kThreads, PER_SM) chunk_delta_kernel(const DeltaRule a) {
  US_PDL_PROLOGUE();
  using St = Stage<DP, CHANNEL>;
  constexpr int kOwn = DP / kSplit, NJ = kOwn / 16;   // channels of a warp, in pairs of eight-wide tiles
  extern __shared__ __align__(128) unsigned char sm[];
  __shared__ __align__(16) Exchange exchange;
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
  if (tid >= kCompute) {
    Feeder<DP, CHANNEL> feed(a, tid - kCompute, start, s, T, h, hk, col0);
    float* out = a.out + ((long long)start * a.H + h) * a.V;
    feed.load(0);
#pragma unroll 1
    for (int ch = 0; ch <= chunks; ++ch) {
      if (ch < chunks) {
        if (ch >= 2) bar_sync(kEmptyBar + (ch & 1), kThreads);
        feed.store(sm + (ch & 1) * St::kBytes);
        bar_arrive(kFullBar + (ch & 1), kThreads);
        if (ch + 1 < chunks) feed.load(ch + 1);
      }
      if (ch == 0) continue;
      bar_sync(kWritesBar + ((ch - 1) & 1) * (kCompute / 32) + warp - kCompute / 32, 64);
      feed.read_out(sm + ((ch - 1) & 1) * St::kBytes, exchange, ch - 1, out);
    }
    return;
  }
  const int tile = warp / kSplit, half = warp % kSplit, r = lane >> 2, i = lane & 3;
  const int cl = tile * 16 + r, col = col0 + cl, dbase = half * kOwn;
  float* Sg = a.state + ((long long)slot * a.H + h) * a.D * a.V;
  const bool fresh = a.pos && a.pos[start] == 0;
  // S^T: tile (j, e) has channels 16 j + 8 e .. of the warp's; a lane's are 2 i and 2 i + 1 of them
  Acc S[NJ][2];
#pragma unroll
  for (int j = 0; j < NJ; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int d = dbase + 16 * j + 8 * e + 2 * i, v = col + c * 8;
        const bool in = !fresh && v < a.V;
        const float* p = Sg + (long long)d * a.V + v;
        S[j][e][c] = pack2(in && d < a.D ? p[0] : 0.f, in && d + 1 < a.D ? p[a.V] : 0.f);
      }
  const uint32_t base0 = (uint32_t)__cvta_generic_to_shared(sm);
  // places of a lane's rows: [n = token][k = channel] operands, [k = token][n = channel] ones, M
  const uint32_t at_x = ((lane & 7) + (lane >> 4) * 8) * St::kRow + (dbase + ((lane >> 3) & 1) * 8) * 2;
  const uint32_t at_s = St::kKr + (lane & 15) * St::kRow + (dbase + (lane >> 4) * 8) * 2;
  const uint32_t at_m = St::kCoefs + ((lane & 7) + (lane >> 4) * 8) * St::kCoefRow + ((lane >> 3) & 1) * 16;
#pragma unroll 1
  for (int ch = 0; ch < chunks; ++ch) {
    bar_sync(kFullBar + (ch & 1), kThreads);
    const unsigned char* base = sm + (ch & 1) * St::kBytes;
    const uint32_t addr = base0 + (ch & 1) * St::kBytes;
    // what keys (tiles 0, 1) and queries (2, 3) see of S0, over this warp's channels
    Acc x[4];
    float low[4][4];
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const Parts sp(S[j][0], S[j][1]);
      float y[4][4];
      products(j == 0, y, low, sp, [&](Tiles& b, int p) {
#pragma unroll
        for (int w = 0; w < 2; ++w) us::ldsm4(b[w], addr + at_x + w * St::kQ + p * St::kPart + j * 32);
      });
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const f2 z = pack2(y[n][2 * c], y[n][2 * c + 1]);
          x[n][c] = j ? add2(x[n][c], z) : z;
        }
    }
    float4(*mine)[32] = exchange[ch & 1][tile][half];
    float4(*other)[32] = exchange[ch & 1][tile][half ^ 1];
#pragma unroll
    for (int n = 0; n < 4; ++n) {
#pragma unroll
      for (int c = 0; c < 2; ++c) x[n][c] = add2(x[n][c], pack2(low[n][2 * c], low[n][2 * c + 1]));
      mine[n][lane] = make_float4(lo2(x[n][0]), hi2(x[n][0]), lo2(x[n][1]), hi2(x[n][1]));
    }
    const float* v = reinterpret_cast<const float*>(base + St::kV);
    const float* vec = reinterpret_cast<const float*>(base + St::kVec);
    const float* decay = reinterpret_cast<const float*>(base + St::kAll);
    f2 beta[2], rest[2];                              // beta_t, R_t16 of tokens 2 i, 2 i + 1 of eight
    Acc w[2], u[2];
    uint32_t m[3][4];
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      beta[n] = *reinterpret_cast<const f2*>(vec + n * 8 + 2 * i);
      rest[n] = CHANNEL ? 0 : *reinterpret_cast<const f2*>(decay + kChunk + n * 8 + 2 * i);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const float* at = v + (n * 8 + 2 * i) * St::kVp + cl + c * 8;
        w[n][c] = pack2(at[0], at[St::kVp]);
      }
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) us::ldsm4(m[q], addr + at_m + q * St::kCoefPart);
    bar_sync(kTileBar + tile, 32 * kSplit);
    // U = M (V - P X)
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const float4 y = other[n][lane];
      const f2 minus = CHANNEL ? pack2(-1.f, -1.f) : mul2(*reinterpret_cast<const f2*>(decay + n * 8 + 2 * i), pack2(-1.f, -1.f));
      w[n][0] = fma2(minus, add2(x[n][0], pack2(y.x, y.y)), w[n][0]);
      w[n][1] = fma2(minus, add2(x[n][1], pack2(y.z, y.w)), w[n][1]);
    }
    {
      const Parts wp(w[0], w[1]);
      float a0[2][4], a1[2][4], a2[2][4];
#pragma unroll
      for (int n = 0; n < 2; ++n) mma_first(a2[n], wp.p[0], m[2][n * 2], m[2][n * 2 + 1]);
#pragma unroll
      for (int n = 0; n < 2; ++n) mma_first(a1[n], wp.p[0], m[1][n * 2], m[1][n * 2 + 1]);
#pragma unroll
      for (int n = 0; n < 2; ++n) mma_first(a0[n], wp.p[0], m[0][n * 2], m[0][n * 2 + 1]);
#pragma unroll
      for (int n = 0; n < 2; ++n) mma(a2[n], wp.p[1], m[1][n * 2], m[1][n * 2 + 1]);
#pragma unroll
      for (int n = 0; n < 2; ++n) mma(a1[n], wp.p[1], m[0][n * 2], m[0][n * 2 + 1]);
#pragma unroll
      for (int n = 0; n < 2; ++n) mma(a2[n], wp.p[2], m[0][n * 2], m[0][n * 2 + 1]);
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const f2 sum = add2(pack2(a1[n][2 * c], a1[n][2 * c + 1]), pack2(a2[n][2 * c], a2[n][2 * c + 1]));
          u[n][c] = fma2(beta[n], w[n][c], add2(pack2(a0[n][2 * c], a0[n][2 * c + 1]), sum));
        }
    }
    const bool finite = all_finite(u[0], u[1]);
    auto hand_on = [&](const Acc(&z)[2]) {
#pragma unroll
      for (int n = 0; n < 2; ++n) other[n][lane] = make_float4(lo2(z[n][0]), hi2(z[n][0]), lo2(z[n][1]), hi2(z[n][1]));
    };
    if (__builtin_expect(!finite, 0)) {               // sums over the tokens up to each one only
      hand_on(w);
      __syncwarp();
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int t = n * 8 + 2 * i;
          u[n][c] = pack2(row_sum<St>(base, 0, t, other, r + c * 8), row_sum<St>(base, 0, t + 1, other, r + c * 8));
        }
      __syncwarp();
    }
    hand_on(u);
    bar_arrive(kWritesBar + (ch & 1) * (kCompute / 32) + warp, 64);
    // S' = P_16 S0 + (R K)^T U
    if (__builtin_expect(finite, 1)) {
      // The last four tokens, which carry most of a state that decays fast, on the FP32 units: beside them the tensor
      // cores' sums would cut more of the others off.
      f2 last[kLast][2];
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          if (!CHANNEL) u[n][c] = mul2(u[n][c], rest[n]);
          if (n == 1) {
#pragma unroll
            for (int t = 0; t < kLast; ++t) {
              const float z = __shfl_sync(0xffffffffu, (t & 1) ? hi2(u[1][c]) : lo2(u[1][c]), (lane & ~3) | (2 + (t >> 1)));
              last[t][c] = pack2(z, z);
            }
            if (i >= 2) u[1][c] = 0;
          }
        }
      const Parts up(u[0], u[1]);
      const float* tail = reinterpret_cast<const float*>(base + St::kTail) + dbase + 4 * i;
      const float all = CHANNEL ? 0.f : decay[kChunk - 1];
#pragma unroll
      for (int j = 0; j < NJ; j += 2) {               // two sixteens of channels
        float y[4][4];
        products(true, y, low, up, [&](Tiles& b, int q) {
#pragma unroll
          for (int f = 0; f < 2; ++f) us::ldsm4t(b[f], addr + at_s + q * St::kPart + (j + f) * 32);
        });
#pragma unroll
        for (int f = 0; f < 2; ++f) {
          f2 k[kLast][2];                             // a lane's channels of both tiles
#pragma unroll
          for (int t = 0; t < kLast; ++t) lds_vec(k[t], tail + t * DP + 16 * (j + f));
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int n = 2 * f + e;
            Acc& x0 = S[j + f][e];
            const f2 g = CHANNEL ? *reinterpret_cast<const f2*>(decay + dbase + 16 * (j + f) + 8 * e + 2 * i) : pack2(all, all);
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              x0[c] = add2(fma2(x0[c], g, pack2(low[n][2 * c], low[n][2 * c + 1])), pack2(y[n][2 * c], y[n][2 * c + 1]));
#pragma unroll
              for (int t = 0; t < kLast; ++t) x0[c] = fma2(k[t][e], last[t][c], x0[c]);
            }
          }
        }
      }
    } else {
      __syncwarp();
      const int n = min(kChunk, T - ch * kChunk);
#pragma unroll
      for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const int d = dbase + 16 * j + 8 * e + 2 * i;
            f2 sum = mul2(S[j][e][c], CHANNEL ? *reinterpret_cast<const f2*>(decay + d)
                                              : pack2(decay[kChunk - 1], decay[kChunk - 1]));
#pragma unroll 1
            for (int t = 0; t < n; ++t) {
              const unsigned char* k = base + St::kKr + t * St::kRow + d * 2;
              const float z = entry(other, r + c * 8, t) * (CHANNEL ? 1.f : decay[kChunk + t]);
              sum = fma2(pack2(whole(k, St::kPart), whole(k + 2, St::kPart)), pack2(z, z), sum);
            }
            S[j][e][c] = sum;
          }
    }
    if (ch + 2 < chunks) bar_arrive(kEmptyBar + (ch & 1), kThreads);
  }
#pragma unroll
  for (int j = 0; j < NJ; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int d = dbase + 16 * j + 8 * e + 2 * i, v = col + c * 8;
        float* p = Sg + (long long)d * a.V + v;
        if (v < a.V && d < a.D) p[0] = lo2(S[j][e][c]);
        if (v < a.V && d + 1 < a.D) p[a.V] = hi2(S[j][e][c]);
      }
}

template <int DP, bool CHANNEL, int PER_SM>
int launch(const DeltaRule& a, dim3 grid, int smem, cudaStream_t stream) {
  US_CUDA_CHECK((us::allow_shared<chunk_delta_kernel<DP, CHANNEL, PER_SM>>(smem)));
  US_CUDA_CHECK(us::launch_pdl(chunk_delta_kernel<DP, CHANNEL, PER_SM>, grid, dim3(kThreads), smem, stream, a));
  return US_OK;
}

template <int DP, bool CHANNEL>
int launch(const DeltaRule& a, cudaStream_t stream) {
  constexpr int need = 2 * Stage<DP, CHANNEL>::kBytes;
  constexpr int alone = need > 110 * 1024 ? need : 110 * 1024;      // shared memory that one CTA per SM has
  int sms = 0;
  US_CUDA_CHECK(us::sm_count(&sms));
  // CTAs that are launched while the kernel before still runs would be packed two to an SM where it
  // leaves room: with fewer CTAs than SMs each asks for more shared memory than half an SM has, and may have more
  // registers (4093 rows, 32 heads of 128 x 128: 128 registers 587 us, 204 531)
  const dim3 grid(us::ceil_div(a.V, kCols), a.H, a.B);
  if ((long long)grid.x * grid.y * grid.z <= sms) return launch<DP, CHANNEL, 1>(a, grid, alone, stream);
  return launch<DP, CHANNEL, (DP > 128 ? 1 : 2)>(a, grid, need, stream);
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
