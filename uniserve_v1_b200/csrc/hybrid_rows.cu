// What stands between the products of the hybrid decoder (bf16 stream, FP32 norm weights), one launch each:
//
//   hybrid_rows   x += sublayer output (rows, or the weighted sum of a token's expert rows, plus shared-expert rows
//                 times a sigmoid); y = x rsqrt(mean(x^2) + eps) w; optionally the dot of y with the shared expert's
//                 gate vector
//   hybrid_heads  per-head norm and half-split rotation of queries and keys of a fused projection, values copied
//   hybrid_gate   rows times the sigmoid of a gate that is interleaved with the queries, head by head
//
// All are bound by memory.  Before, PyTorch's elementwise kernels ran them: eleven passes for a norm with its residual
// (4093 rows of 2048: 89 us), 21 for a layer's queries and keys (380 us), five for an expert sum.  Arithmetic is FP32, rounded
// where those passes stored their results.
#include "include/us_common.cuh"

namespace {

constexpr int kRowThreads = 256;

struct RowsArgs {
  const __nv_bfloat16 *x, *add;           // [T, H]; add null: none
  const __nv_bfloat16 *routed;            // [R, H] expert rows, with perm / weights [T, top]
  const int* perm;
  const float* weights;
  const __nv_bfloat16* shared;            // [T, H], times sigmoid(shared_gate[t])
  const float* shared_gate;
  const float* w;                         // [H]
  const __nv_bfloat16* gate_w;            // [H] or null
  __nv_bfloat16 *out, *y;                 // the new stream (null: x stands), its norm
  float* gate;                            // [T]
  long long ldx, ldadd;
  int H, top;
  float eps;
};

// One CTA per row, the row in registers (NV x 8 values a thread): x and the sublayer's rows are read once.
template <int NV>
__global__ void __launch_bounds__(kRowThreads) hybrid_rows_kernel(const RowsArgs a) {
  US_PDL_PROLOGUE();
  __shared__ float scratch[33];
  const long long row = blockIdx.x;
  const int nvec = a.H >> 3;
  const float sg = a.shared ? 1.f / (1.f + expf(-a.shared_gate[row])) : 0.f;
  float v[NV][8], ss = 0.f;
#pragma unroll
  for (int n = 0; n < NV; ++n) {
    const int c = threadIdx.x + n * kRowThreads;
    if (c >= nvec) break;
    us::Pack16 p;
    p.u = *reinterpret_cast<const uint4*>(a.x + row * a.ldx + c * 8);
    float s[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) s[i] = 0.f;
    if (a.add) {
      us::Pack16 q;
      q.u = *reinterpret_cast<const uint4*>(a.add + row * a.ldadd + c * 8);
#pragma unroll
      for (int i = 0; i < 8; ++i) s[i] = us::bf2f(q.b[i]);
    }
    if (a.routed) {
      for (int j = 0; j < a.top; ++j) {
        const int at = a.perm[row * a.top + j];
        if (at < 0) continue;
        const float wt = a.weights[row * a.top + j];
        us::Pack16 q;
        q.u = *reinterpret_cast<const uint4*>(a.routed + (long long)at * a.H + c * 8);
#pragma unroll
        for (int i = 0; i < 8; ++i) s[i] += wt * us::bf2f(q.b[i]);
      }
    }
    // rounded where the model's formulas round: the experts' sum, the shared rows, their sum
#pragma unroll
    for (int i = 0; i < 8; ++i) s[i] = us::bf2f(us::f2bf(s[i]));
    if (a.shared) {
      us::Pack16 q;
      q.u = *reinterpret_cast<const uint4*>(a.shared + row * a.H + c * 8);
#pragma unroll
      for (int i = 0; i < 8; ++i) s[i] = us::bf2f(us::f2bf(s[i] + us::bf2f(us::f2bf(sg * us::bf2f(q.b[i])))));
    }
    us::Pack16 o;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      o.b[i] = us::f2bf(us::bf2f(p.b[i]) + s[i]);
      v[n][i] = us::bf2f(o.b[i]);                      // the norm sees the stream as it is stored
      ss += v[n][i] * v[n][i];
    }
    if (a.out) *reinterpret_cast<uint4*>(a.out + row * a.H + c * 8) = o.u;
  }
  const float inv = rsqrtf(us::block_sum(ss, scratch) / (float)a.H + a.eps);
  float dot = 0.f;
#pragma unroll
  for (int n = 0; n < NV; ++n) {
    const int c = threadIdx.x + n * kRowThreads;
    if (c >= nvec) break;
    const float4 w0 = *reinterpret_cast<const float4*>(a.w + c * 8), w1 = *reinterpret_cast<const float4*>(a.w + c * 8 + 4);
    const float w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
    us::Pack16 o;
#pragma unroll
    for (int i = 0; i < 8; ++i) o.b[i] = us::f2bf(v[n][i] * inv * w[i]);
    *reinterpret_cast<uint4*>(a.y + row * a.H + c * 8) = o.u;
    if (a.gate_w) {
      us::Pack16 q;
      q.u = *reinterpret_cast<const uint4*>(a.gate_w + c * 8);
#pragma unroll
      for (int i = 0; i < 8; ++i) dot = fmaf(us::bf2f(o.b[i]), us::bf2f(q.b[i]), dot);
    }
  }
  if (a.gate_w) {
    dot = us::block_sum(dot, scratch);
    if (threadIdx.x == 0) a.gate[row] = dot;
  }
}

constexpr int kHeadWarps = 8, kMaxD = 256;

struct HeadsArgs {
  const __nv_bfloat16* proj;              // [T, ld]: Hq (query, gate) pairs of D, then Hk keys, then Hk values
  const float *qw, *kw;                   // [D]
  const float* inv_freq;                  // [rot / 2]
  __nv_bfloat16 *q, *k, *v;               // [T, Hq, D], [T, Hk, D] x 2
  long long ld;
  int pos0, Hq, Hk, D, rot;
  float eps;
};

// A CTA per row (its angles once), a warp per head; a lane has channels lane * 4 .. and, past 128, 128 + lane * 4 ..
__global__ void __launch_bounds__(kHeadWarps * 32) hybrid_heads_kernel(const HeadsArgs a) {
  US_PDL_PROLOGUE();
  __shared__ float2 turn[kMaxD / 2];
  __shared__ __align__(16) float rows[kHeadWarps][kMaxD];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, half = a.rot >> 1;
  const long long t = blockIdx.x;
  if ((int)threadIdx.x < half) {
    float sn, cs;
    sincosf((float)(a.pos0 + t) * a.inv_freq[threadIdx.x], &sn, &cs);
    turn[threadIdx.x] = make_float2(cs, sn);
  }
  __syncthreads();
  const __nv_bfloat16* p = a.proj + t * a.ld;
  float* buf = rows[warp];
  for (int h = warp; h < a.Hq + 2 * a.Hk; h += kHeadWarps) {
    const bool is_q = h < a.Hq;
    const __nv_bfloat16* src = p + (is_q ? (long long)h * 2 * a.D : (long long)(h + a.Hq) * a.D);
    if (h >= a.Hq + a.Hk) {
      __nv_bfloat16* dst = a.v + (t * a.Hk + h - a.Hq - a.Hk) * a.D;
      for (int c = lane * 4; c < a.D; c += 128) *reinterpret_cast<uint2*>(dst + c) = *reinterpret_cast<const uint2*>(src + c);
      continue;
    }
    float x[2][4], ss = 0.f;
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const int c = lane * 4 + n * 128;
      if (c >= a.D) break;
      us::Pack8 o;
      o.u = *reinterpret_cast<const uint2*>(src + c);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        x[n][i] = us::bf2f(o.b[i]);
        ss += x[n][i] * x[n][i];
      }
    }
    const float inv = rsqrtf(us::warp_sum(ss) / (float)a.D + a.eps);
    const float* w = is_q ? a.qw : a.kw;
    __syncwarp();                                      // the head before has been read
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const int c = lane * 4 + n * 128;
      if (c >= a.D) break;
      const float4 g = *reinterpret_cast<const float4*>(w + c);
      *reinterpret_cast<float4*>(buf + c) = make_float4(x[n][0] * inv * g.x, x[n][1] * inv * g.y, x[n][2] * inv * g.z,
                                                        x[n][3] * inv * g.w);
    }
    __syncwarp();
    __nv_bfloat16* dst = is_q ? a.q + (t * a.Hq + h) * a.D : a.k + (t * a.Hk + h - a.Hq) * a.D;
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const int c = lane * 4 + n * 128;
      if (c >= a.D) break;
      us::Pack8 o;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int e = c + i;
        float r = buf[e];
        if (e < half) r = r * turn[e].x - buf[e + half] * turn[e].y;
        else if (e < a.rot) r = r * turn[e - half].x + buf[e - half] * turn[e - half].y;
        o.b[i] = us::f2bf(r);
      }
      *reinterpret_cast<uint2*>(dst + c) = o.u;
    }
  }
}

__global__ void __launch_bounds__(256)
hybrid_gate_kernel(const __nv_bfloat16* __restrict__ att, const __nv_bfloat16* __restrict__ gates, long long ld,
                   __nv_bfloat16* __restrict__ out, long long vecs, int row_vecs, int D) {
  US_PDL_PROLOGUE();
  for (long long e = blockIdx.x * 256ll + threadIdx.x; e < vecs; e += 256ll * gridDim.x) {
    const long long t = e / row_vecs;
    const int c = (int)(e - t * row_vecs) * 8, h = c / D;
    us::Pack16 x, g, o;
    x.u = *reinterpret_cast<const uint4*>(att + e * 8);
    g.u = *reinterpret_cast<const uint4*>(gates + t * ld + (2 * h + 1) * D + (c - h * D));
#pragma unroll
    for (int i = 0; i < 8; ++i) o.b[i] = us::f2bf(us::bf2f(x.b[i]) / (1.f + expf(-us::bf2f(g.b[i]))));
    *reinterpret_cast<uint4*>(out + e * 8) = o.u;
  }
}

inline bool on16(const void* p) { return ((uintptr_t)p % 16) == 0; }

}  // namespace

// H a multiple of 8, at most 8192; every pointer on 16 bytes.
US_API int us_hybrid_rows(const void* x, long long ldx, const void* add, long long ldadd, const void* routed,
                          const int* perm, const float* weights, int top, const void* shared, const float* shared_gate,
                          const float* w, const void* gate_w, void* out, void* y, float* gate, int T, int H, float eps,
                          void* stream_) {
  US_REQUIRE(x && w && y && T >= 0 && H >= 8 && H % 8 == 0 && H <= 8192 && ldx % 8 == 0 && ldadd % 8 == 0);
  US_REQUIRE((!routed || (perm && weights && top >= 1)) && (!shared || shared_gate) && (!gate_w || gate));
  US_REQUIRE(on16(x) && on16(add) && on16(routed) && on16(shared) && on16(w) && on16(gate_w) && on16(out) && on16(y));
  if (T == 0) return US_OK;
  RowsArgs a{(const __nv_bfloat16*)x, (const __nv_bfloat16*)add, (const __nv_bfloat16*)routed, perm, weights,
             (const __nv_bfloat16*)shared, shared_gate, w, (const __nv_bfloat16*)gate_w, (__nv_bfloat16*)out,
             (__nv_bfloat16*)y, gate, ldx, ldadd, H, top, eps};
  const int per = us::ceil_div(H / 8, kRowThreads);
  auto kernel = per == 1 ? hybrid_rows_kernel<1> : per == 2 ? hybrid_rows_kernel<2> : hybrid_rows_kernel<4>;
  US_CUDA_CHECK(us::launch_pdl(kernel, dim3(T), dim3(kRowThreads), 0, (cudaStream_t)stream_, a));
  return US_OK;
}

// D a multiple of 8, at most 256; rot even, at most D.
US_API int us_hybrid_heads(const void* proj, long long ld, const float* qw, const float* kw, const float* inv_freq,
                           void* q, void* k, void* v, int T, int pos0, int Hq, int Hk, int D, int rot, float eps,
                           void* stream_) {
  US_REQUIRE(proj && qw && kw && (inv_freq || rot == 0) && q && k && v && T >= 0 && Hq >= 1 && Hk >= 1 && ld % 8 == 0);
  US_REQUIRE(D >= 8 && D % 8 == 0 && D <= kMaxD && rot >= 0 && rot <= D && rot % 2 == 0);
  US_REQUIRE(on16(proj) && on16(qw) && on16(kw) && on16(q) && on16(k) && on16(v));
  if (T == 0) return US_OK;
  HeadsArgs a{(const __nv_bfloat16*)proj, qw, kw, inv_freq, (__nv_bfloat16*)q, (__nv_bfloat16*)k, (__nv_bfloat16*)v, ld,
              pos0, Hq, Hk, D, rot, eps};
  US_CUDA_CHECK(us::launch_pdl(hybrid_heads_kernel, dim3(T), dim3(kHeadWarps * 32), 0, (cudaStream_t)stream_, a));
  return US_OK;
}

US_API int us_hybrid_gate(const void* att, const void* proj, long long ld, void* out, int T, int Hq, int D,
                          void* stream_) {
  US_REQUIRE(att && proj && out && T >= 0 && Hq >= 1 && D >= 8 && D % 8 == 0 && ld % 8 == 0);
  US_REQUIRE(on16(att) && on16(proj) && on16(out));
  if (T == 0) return US_OK;
  const long long vecs = (long long)T * Hq * D / 8, blocks = (vecs + 255) / 256;
  US_CUDA_CHECK(us::launch_pdl(hybrid_gate_kernel, dim3((unsigned)(blocks < 148 * 16 ? blocks : 148 * 16)), dim3(256), 0,
                               (cudaStream_t)stream_, (const __nv_bfloat16*)att, (const __nv_bfloat16*)proj, ld,
                               (__nv_bfloat16*)out, vecs, Hq * D / 8, D));
  return US_OK;
}
