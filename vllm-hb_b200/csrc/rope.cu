// Rotary position embedding.
//
// hb_rope: one CTA per token.  The token's cos/sin row is computed once in f32 from
// positions[t] * inv_freq[i], rounded to the tensor dtype (apply_rope casts its tables
// with to_dtype, src/engine/arch/llama_tp.rs:132-133) and shared by all q and k heads
// of the token; every thread then rotates 128-bit vector pairs (d, d + head_dim/2).
// q and k carry their own head counts, so GQA is handled (the reference's fused
// rope_inplace kernel indexes k with the q head count, kernels/rope.cu:83).
//
// hb_rope_cos_sin: the calling convention of rope_single_{f32,f16}
// (kernels/rope.cu:19-63): tables pre-sliced by the caller, position = token % seq_len.
#include "common.h"

namespace hb {

constexpr int kRopeThreads = 128;
constexpr int kMaxHalf = 256;  // head_dim <= 512

template <typename T>
__global__ void __launch_bounds__(kRopeThreads)
rope_kernel(T* __restrict__ q, T* __restrict__ k, const int32_t* __restrict__ positions,
            const float* __restrict__ inv_freq, int nq, int nkv, int head_dim) {
  __shared__ float s_cos[kMaxHalf];
  __shared__ float s_sin[kMaxHalf];
  const int64_t t = blockIdx.x;
  const int half = head_dim >> 1;
  const float pos = (float)positions[t];
  for (int i = threadIdx.x; i < half; i += kRopeThreads) {
    const float f = pos * inv_freq[i];
    float s, c;
    sincosf(f, &s, &c);
    s_cos[i] = to_f32<T>(from_f32<T>(c));
    s_sin[i] = to_f32<T>(from_f32<T>(s));
  }
  __syncthreads();

  constexpr int N = Vec16<T>::N;
  const int heads = nq + (k ? nkv : 0);
  if (half % N == 0) {
    const int vph = half / N;  // vector pairs per head
    for (int idx = threadIdx.x; idx < heads * vph; idx += kRopeThreads) {
      const int h = idx / vph, v = idx % vph;
      T* base = (h < nq) ? q + (t * nq + h) * head_dim : k + (t * nkv + (h - nq)) * head_dim;
      Vec16<T> a, b;
      a.load(base + v * N);
      b.load(base + half + v * N);
      float x1[N], x2[N], o1[N], o2[N];
      a.unpack(x1);
      b.unpack(x2);
#pragma unroll
      for (int j = 0; j < N; ++j) {
        const float c = s_cos[v * N + j], s = s_sin[v * N + j];
        o1[j] = x1[j] * c - x2[j] * s;
        o2[j] = x1[j] * s + x2[j] * c;
      }
      a.pack(o1);
      b.pack(o2);
      a.store(base + v * N);
      b.store(base + half + v * N);
    }
  } else {
    for (int idx = threadIdx.x; idx < heads * half; idx += kRopeThreads) {
      const int h = idx / half, d = idx % half;
      T* base = (h < nq) ? q + (t * nq + h) * head_dim : k + (t * nkv + (h - nq)) * head_dim;
      const float x1 = to_f32<T>(base[d]), x2 = to_f32<T>(base[d + half]);
      const float c = s_cos[d], s = s_sin[d];
      base[d] = from_f32<T>(x1 * c - x2 * s);
      base[d + half] = from_f32<T>(x1 * s + x2 * c);
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(kRopeThreads)
rope_cos_sin_kernel(T* __restrict__ out, const T* __restrict__ x, const T* __restrict__ cos_t,
                    const T* __restrict__ sin_t, int64_t seq_len, int head_dim) {
  const int64_t token = blockIdx.x;  // over batch*heads*seq
  const int half = head_dim >> 1;
  const int64_t t = token % seq_len;
  const T* xi = x + token * head_dim;
  T* yo = out + token * head_dim;
  for (int d = threadIdx.x; d < half; d += kRopeThreads) {
    const float x0 = to_f32<T>(xi[d]), x1 = to_f32<T>(xi[d + half]);
    const float c = to_f32<T>(cos_t[t * half + d]), s = to_f32<T>(sin_t[t * half + d]);
    yo[d] = from_f32<T>(x0 * c - x1 * s);
    yo[d + half] = from_f32<T>(x0 * s + x1 * c);
  }
}

// Rows of 16-byte vectors, of q and then of k (rows_k may be 0): a thread rotates one vector pair
// (d, d + head_dim / 2).  One launch for both: at one token the launches are what it costs.
template <typename T>
__global__ void __launch_bounds__(256)
rope_cos_sin_vec_kernel(T* __restrict__ out_q, const T* __restrict__ q, int64_t rows_q, T* __restrict__ out_k, const T* __restrict__ k,
                        int64_t rows_k, const T* __restrict__ cos_t, const T* __restrict__ sin_t, int64_t seq_len, int vph) {
  constexpr int N = Vec16<T>::N;
  const int64_t idx = (int64_t)blockIdx.x * 256 + threadIdx.x, r = idx / vph;
  const int v = (int)(idx % vph), half = vph * N;
  if (r >= rows_q + rows_k) return;
  const bool is_q = r < rows_q;
  const int64_t row = is_q ? r : r - rows_q, t = row % seq_len;
  const T* x = (is_q ? q : k) + row * 2 * half + v * N;
  T* y = (is_q ? out_q : out_k) + row * 2 * half + v * N;
  Vec16<T> a, b, cv, sv;
  a.load(x);
  b.load(x + half);
  cv.load(cos_t + t * half + v * N);
  sv.load(sin_t + t * half + v * N);
  float x0[N], x1[N], c[N], s[N], o0[N], o1[N];
  a.unpack(x0);
  b.unpack(x1);
  cv.unpack(c);
  sv.unpack(s);
#pragma unroll
  for (int j = 0; j < N; ++j) {
    o0[j] = x0[j] * c[j] - x1[j] * s[j];
    o1[j] = x0[j] * s[j] + x1[j] * c[j];
  }
  a.pack(o0);
  b.pack(o1);
  a.store(y);
  b.store(y + half);
}

// Whether every row of `x` and `out` is made of 16-byte vectors.
static bool rope_vectors(const void* out, const void* x, const void* cos_t, const void* sin_t, int head_dim, hb_dtype dtype) {
  const uintptr_t all = reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(cos_t) |
                        reinterpret_cast<uintptr_t>(sin_t);
  return (all & 15) == 0 && (head_dim / 2 * dtype_size(dtype)) % 16 == 0;
}

static int rope_vec(cudaStream_t st, void* out_q, const void* q, int64_t rows_q, void* out_k, const void* k, int64_t rows_k,
                    const void* cos_t, const void* sin_t, int64_t seq_len, int head_dim, hb_dtype dtype) {
  HB_DISPATCH_DTYPE(dtype, T, {
    const int vph = head_dim / 2 / Vec16<T>::N;
    const int64_t ctas = ((rows_q + rows_k) * vph + 255) / 256;
    rope_cos_sin_vec_kernel<T><<<(unsigned)ctas, 256, 0, st>>>((T*)out_q, (const T*)q, rows_q, (T*)out_k, (const T*)k, rows_k,
                                                               (const T*)cos_t, (const T*)sin_t, seq_len, vph);
  });
  HB_LAUNCH_CHECK();
  return HB_OK;
}

}  // namespace hb

extern "C" {

int hb_rope_inv_freq(float theta, int head_dim, float* out) {
  HB_CHECK_ARG(out && head_dim > 0 && head_dim % 2 == 0, "hb_rope_inv_freq: bad head_dim %d",
               head_dim);
  const int half = head_dim / 2;
  for (int i = 0; i < half; ++i)
    out[i] = 1.0f / powf(theta, 2.0f * (float)i / (float)head_dim);
  return HB_OK;
}

int hb_rope(void* stream, void* q, void* k, const int32_t* positions, const float* inv_freq,
            int64_t n_tokens, int n_q_heads, int n_kv_heads, int head_dim, hb_dtype dtype) {
  HB_CHECK_ARG(q && positions && inv_freq, "hb_rope: null pointer");
  HB_CHECK_ARG(head_dim > 0 && head_dim % 2 == 0 && head_dim / 2 <= hb::kMaxHalf,
               "hb_rope: head_dim %d must be even and <= %d", head_dim, 2 * hb::kMaxHalf);
  HB_CHECK_ARG(n_q_heads > 0 && (!k || n_kv_heads > 0), "hb_rope: bad head counts");
  HB_CHECK_ARG(n_tokens >= 0 && n_tokens < (1ll << 31), "hb_rope: bad n_tokens");
  if (n_tokens == 0) return HB_OK;
  HB_CHECK_ARG((reinterpret_cast<uintptr_t>(q) & 15) == 0 &&
                   (reinterpret_cast<uintptr_t>(k) & 15) == 0,
               "hb_rope: q and k must be 16-byte aligned");
  HB_DISPATCH_DTYPE(dtype, T, {
    const bool vec_ok = ((head_dim / 2) % hb::Vec16<T>::N == 0);
    (void)vec_ok;
    hb::rope_kernel<T><<<(unsigned)n_tokens, hb::kRopeThreads, 0, (cudaStream_t)stream>>>(
        (T*)q, (T*)k, positions, inv_freq, n_q_heads, n_kv_heads, head_dim);
  });
  HB_LAUNCH_CHECK();
  return HB_OK;
}

int hb_rope_cos_sin(void* stream, void* out, const void* x, const void* cos_table,
                    const void* sin_table, int64_t batch_heads, int64_t seq_len, int head_dim,
                    hb_dtype dtype) {
  HB_CHECK_ARG(out && x && cos_table && sin_table, "hb_rope_cos_sin: null pointer");
  HB_CHECK_ARG(head_dim > 0 && head_dim % 2 == 0, "hb_rope_cos_sin: head_dim must be even");
  HB_CHECK_ARG(batch_heads >= 0 && seq_len > 0 && batch_heads * seq_len < (1ll << 31),
               "hb_rope_cos_sin: bad shape");
  if (batch_heads == 0) return HB_OK;
  if (hb::dtype_valid(dtype) && hb::rope_vectors(out, x, cos_table, sin_table, head_dim, dtype))
    return hb::rope_vec((cudaStream_t)stream, out, x, batch_heads * seq_len, nullptr, nullptr, 0, cos_table, sin_table, seq_len,
                        head_dim, dtype);
  HB_DISPATCH_DTYPE(dtype, T, {
    hb::rope_cos_sin_kernel<T><<<(unsigned)(batch_heads * seq_len), hb::kRopeThreads, 0,
                                 (cudaStream_t)stream>>>((T*)out, (const T*)x, (const T*)cos_table,
                                                         (const T*)sin_table, seq_len, head_dim);
  });
  HB_LAUNCH_CHECK();
  return HB_OK;
}

int hb_rope_cos_sin_pair(void* stream, void* out_q, const void* q, int64_t batch_heads_q, void* out_k, const void* k,
                         int64_t batch_heads_k, const void* cos_table, const void* sin_table, int64_t seq_len, int head_dim,
                         hb_dtype dtype) {
  HB_CHECK_ARG(out_q && q && out_k && k && cos_table && sin_table, "hb_rope_cos_sin_pair: null pointer");
  HB_CHECK_ARG(head_dim > 0 && head_dim % 2 == 0, "hb_rope_cos_sin_pair: head_dim must be even");
  HB_CHECK_ARG(batch_heads_q >= 0 && batch_heads_k >= 0 && seq_len > 0 && batch_heads_q * seq_len < (1ll << 31) &&
                   batch_heads_k * seq_len < (1ll << 31), "hb_rope_cos_sin_pair: bad shape");
  if (batch_heads_q && batch_heads_k && hb::dtype_valid(dtype) &&
      hb::rope_vectors(out_q, q, cos_table, sin_table, head_dim, dtype) &&
      hb::rope_vectors(out_k, k, cos_table, sin_table, head_dim, dtype))
    return hb::rope_vec((cudaStream_t)stream, out_q, q, batch_heads_q * seq_len, out_k, k, batch_heads_k * seq_len, cos_table,
                        sin_table, seq_len, head_dim, dtype);
  const int rc = hb_rope_cos_sin(stream, out_q, q, cos_table, sin_table, batch_heads_q, seq_len, head_dim, dtype);
  return rc ? rc : hb_rope_cos_sin(stream, out_k, k, cos_table, sin_table, batch_heads_k, seq_len, head_dim, dtype);
}

}  // extern "C"
