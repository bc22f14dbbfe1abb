// Attention of prompt portions on 5th-generation tensor cores (bf16 or f16, head_dim 128, paged pools).
//
// CTA = 128 rows of queries: up to 128 / R consecutive positions of one sequence x the R query heads of a kv
// head.  Per step of 64 keys (four blocks of the pool, by TMA with the 128-byte swizzle):
//   S [128 x 64]   = Q K^T   both operands in shared memory, S in tensor memory
//   P              = 2^(S - m): a thread owns a row, so maximum and sum need no exchange
//   O [128 x 128] += P V     P in tensor memory (operand A), V as it lies ([key][channel], MN-major)
// P is a pair of 16-bit numbers (hi + lo), two products: weights keep 16 bits (f16: 22), as in the tile kernel
// on warp-level products (attention_span_mma.cu).  O is rescaled only when a row's maximum has grown by more
// than 2^8 since m was taken, so hardly ever: until then P may reach 2^8, which changes no relative rounding.
//
//   warps 0-3: softmax, a row per thread     warp 4: TMA producer     warp 5: MMA issuer
//
// S of the next step is issued before O of this one, so that the tensor cores work while the softmax warps
// do; K and V stages are released separately.  256 columns of tensor memory and 97 KB of shared memory: two CTAs
// share an SM.  Every wait is bounded.
//
// Bound: at prompt lengths of a few thousand tokens the chain S -> softmax -> P -> O of one step, as there are
// fewer CTAs than SM places.  Prefill of 2000 tokens in steps of 512 rows, 32 / 8 heads, 8 layers: 9.32 ms with 64-row
// tiles on warp-level products, 8.40 ms with these.
#include <cuda.h>

#include <algorithm>
#include <climits>
#include <mutex>

#include "layered_ops.h"
#include "span_core.cuh"

namespace hb {

namespace {
constexpr int kPromptThreads = 192;
constexpr int kPromptKeys = 64;
constexpr int kPD = 128;                       // head_dim
constexpr uint32_t kPromptQ = 128 * kPD * 2;   // bytes
constexpr uint32_t kPromptTile = kPromptKeys * kPD * 2;
constexpr size_t kPromptSmem = kPromptQ + 4 * kPromptTile + 1024;
constexpr uint32_t kColS = 0, kColO = 64, kColHi = 192, kColLo = 224;
}  // namespace

// D (+)= A * B, A in tensor memory
__device__ __forceinline__ void umma_ts_if(uint32_t e, uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(e)
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// Shared-memory descriptor of an operand whose rows run along K (MN-major), 128-byte swizzle: runs of 64 elements
// along M/N, 8 rows of K per 1024 bytes; lbo: bytes from one run of 64 to the next.
__device__ __forceinline__ uint64_t make_smem_desc_mn(uint32_t saddr, uint32_t lbo) {
  return (make_smem_desc(saddr) & ~((uint64_t)0x3FFF << 16)) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16);
}

template <typename T>
__global__ void __launch_bounds__(kPromptThreads, 2)
prompt_attention_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, const SpanAttention a,
                        const RowRange* __restrict__ tiles) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t s_kfull[2], s_kempty[2], s_vfull[2], s_vempty[2];
  __shared__ __align__(8) uint64_t s_sfull, s_sfree, s_pfull, s_done;
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;
  constexpr bool HALF = std::is_same<T, __half>::value;
  constexpr float kPScale = HALF ? 128.f : 1.f;  // f16: the pair's low part stays above the smallest numbers
  constexpr float kGrow = 8.f;                   // of a maximum, in units of log2, before O is rescaled
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int R = a.heads / a.kv_heads, kvh = blockIdx.y;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u, k_base = base + kPromptQ, v_base = k_base + 2 * kPromptTile;
  uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&s_kfull[i]), 1);
      mbar_init(smem_u32(&s_kempty[i]), 1);
      mbar_init(smem_u32(&s_vfull[i]), 1);
      mbar_init(smem_u32(&s_vempty[i]), 1);
    }
    mbar_init(smem_u32(&s_sfull), 1);
    mbar_init(smem_u32(&s_sfree), 4);
    mbar_init(smem_u32(&s_pfull), 4);
    mbar_init(smem_u32(&s_done), 1);
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 5) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(256) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  pdl_grid_wait();
  const RowRange tile = tiles[gridDim.x - 1 - blockIdx.x];  // later positions see more: they go first
  const int first_pos = a.pos[tile.row0], last_pos = first_pos + tile.n - 1;
  const BlockRuns runs = block_runs(first_pos, last_pos, a);
  const int n_rows = tile.n * R, n_steps = (runs.n + 3) / 4;

  // queries: 16-byte vectors to their swizzled places, two halves of 64 channels; rows that do not exist are zero
  const T* q = (const T*)a.q + (int64_t)kvh * R * kPD;
  for (int i = tid; i < 128 * (kPD / 8); i += kPromptThreads) {
    const int m = i / (kPD / 8), c = i % (kPD / 8);
    uint4 v = make_uint4(0, 0, 0, 0);
    if (m < n_rows) v = *reinterpret_cast<const uint4*>(q + (int64_t)(tile.row0 + m / R) * a.ld_q + (m % R) * kPD + c * 8);
    *reinterpret_cast<uint4*>(gen + (c >> 3) * 16384 + m * 128 + (((c & 7) ^ (m & 7)) << 4)) = v;
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;

  if (warp == 4) {
    // -------------------------------------------------------------- TMA producer
    const uint32_t e = elect_one();
    const int32_t* table = a.tables + (int64_t)tile.seg * a.max_blocks;
    int tab_base = -32, tab = 0;
    bool ok = true;
    int i = 0;
    for (; i < n_steps; ++i) {
      const int s = i & 1;
      const uint32_t par = ((uint32_t)(i >> 1) & 1u) ^ 1u;
      if (i * 4 >= tab_base + 32) {  // the next 32 entries, one per lane
        tab_base = i * 4;
        const int lb = runs.block(min(tab_base + lane, runs.n - 1));  // past the last: any, its keys are masked
        tab = lb < a.max_blocks ? table[lb] : 0;
        if (tab < 0 || tab >= a.num_blocks) tab = 0;  // never outside the pool
      }
      int row[4];
#pragma unroll
      for (int b = 0; b < 4; ++b)
        row[b] = (int)(((int64_t)__shfl_sync(0xffffffffu, tab, i * 4 + b - tab_base) * a.kv_heads + kvh) * kBS);
      ok = mbar_wait(smem_u32(&s_kempty[s]), par, &s_abort);
      if (!ok) break;
      const uint32_t kf = smem_u32(&s_kfull[s]), kd = k_base + s * kPromptTile;
      mbar_expect_tx_if(e, kf, kPromptTile);
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        tma_load_2d_if(e, kd + b * 2048, &tm_k, 0, row[b], kf);
        tma_load_2d_if(e, kd + kPromptTile / 2 + b * 2048, &tm_k, 64, row[b], kf);
      }
      ok = mbar_wait(smem_u32(&s_vempty[s]), par, &s_abort);
      if (!ok) { ++i; break; }
      const uint32_t vf = smem_u32(&s_vfull[s]), vd = v_base + s * kPromptTile;
      mbar_expect_tx_if(e, vf, kPromptTile);
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        tma_load_2d_if(e, vd + b * 2048, &tm_v, 0, row[b], vf);
        tma_load_2d_if(e, vd + kPromptTile / 2 + b * 2048, &tm_v, 64, row[b], vf);
      }
    }
    if (s_abort)  // let the copies that were issued land: a barrier is between phases or completes the open one
      for (int s = 0; s < 2; ++s)
        for (uint64_t* bar : {&s_kfull[s], &s_vfull[s]})
          for (uint32_t n = 0; n < kSpinLimit / 16 && !mbar_try(smem_u32(bar), 0) && !mbar_try(smem_u32(bar), 1); ++n) {
          }
    __syncwarp();
  } else if (warp == 5) {
    // -------------------------------------------------------------- MMA issuer
    const uint32_t e = elect_one();
    const uint32_t id_s = make_idesc<T>(kPromptKeys), id_o = make_idesc<T>(kPD) | (1u << 16);  // V: MN-major
    const uint32_t acc = __shfl_sync(0xffffffffu, tmem, 0);
    bool ok = true;
    auto scores = [&](int i) {
      const uint64_t qd = make_smem_desc(base), kd = make_smem_desc(k_base + (i & 1) * kPromptTile);
#pragma unroll
      for (int k = 0; k < kPD / 16; ++k)  // 16 channels = 32 bytes; the second half of the channels is a tile of its own
        umma_if(e, acc + kColS, qd + (uint64_t)((k >> 2) * (16384 >> 4) + (k & 3) * 2),
                kd + (uint64_t)((k >> 2) * (kPromptTile / 2 >> 4) + (k & 3) * 2), id_s, k > 0 ? 1u : 0u);
      tc_commit_if(e, smem_u32(&s_kempty[i & 1]));
      tc_commit_if(e, smem_u32(&s_sfull));
    };
    ok = mbar_wait(smem_u32(&s_kfull[0]), 0, &s_abort);
    if (ok) {
      tc_fence_after();
      scores(0);
    }
    for (int i = 0; i < n_steps && ok; ++i) {
      if (i + 1 < n_steps) {
        ok = mbar_wait(smem_u32(&s_kfull[(i + 1) & 1]), (uint32_t)((i + 1) >> 1) & 1u, &s_abort) &&
             mbar_wait(smem_u32(&s_sfree), (uint32_t)i & 1u, &s_abort);
        if (!ok) break;
        tc_fence_after();
        scores(i + 1);
      }
      ok = mbar_wait(smem_u32(&s_vfull[i & 1]), (uint32_t)(i >> 1) & 1u, &s_abort) &&
           mbar_wait(smem_u32(&s_pfull), (uint32_t)i & 1u, &s_abort);
      if (!ok) break;
      tc_fence_after();
      const uint64_t vd = make_smem_desc_mn(v_base + (i & 1) * kPromptTile, kPromptTile / 2);
#pragma unroll
      for (int part = 0; part < 2; ++part)
#pragma unroll
        for (int k = 0; k < kPromptKeys / 16; ++k)  // 16 keys: 8 columns of P, 2048 bytes of V
          umma_ts_if(e, acc + kColO, acc + (part ? kColLo : kColHi) + k * 8, vd + (uint64_t)(k * (2048 >> 4)), id_o,
                     (i > 0 || part > 0 || k > 0) ? 1u : 0u);
      tc_commit_if(e, smem_u32(&s_vempty[i & 1]));
      tc_commit_if(e, smem_u32(&s_done));
    }
    __syncwarp();
  } else {
    // -------------------------------------------------------------- softmax, a row per thread
    const int r = warp * 32 + lane, pos = first_pos + r / R, lo = a.first_seen(pos);
    const uint32_t t_lane = tmem + ((uint32_t)(warp * 32) << 16);
    const int warp_first = first_pos + warp * 32 / R, warp_last = min(first_pos + (warp * 32 + 31) / R, last_pos);
    const int warp_lo = a.first_seen(warp_last);
    const float sc = a.scale * kLog2e;
    float m = -INFINITY, l = 0.f;  // m: what the exponentials are taken against, in units of log2
    bool ok = true;
    for (int i = 0; i < n_steps; ++i) {
      ok = mbar_wait(smem_u32(&s_sfull), (uint32_t)i & 1u, &s_abort);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      float s[64];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld16(t_lane + kColS + c * 16, *reinterpret_cast<float(*)[16]>(&s[c * 16]));
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&s_sfree));
      float mx = -INFINITY;
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int vb = i * 4 + b, key = vb < runs.n ? runs.block(vb) * kBS : INT_MAX - kBS;
        if (vb < runs.n && all_visible(key, warp_first, warp_lo, a.keep_first)) {
#pragma unroll
          for (int j = 0; j < 16; ++j) s[b * 16 + j] *= sc;
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) s[b * 16 + j] = visible(key + j, pos, lo, a.keep_first) ? s[b * 16 + j] * sc : -INFINITY;
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) mx = fmaxf(mx, s[b * 16 + j]);
      }
      if (i > 0) {  // P and O of the step before are done with
        ok = mbar_wait(smem_u32(&s_done), (uint32_t)(i - 1) & 1u, &s_abort);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
      }
      const bool grow = mx > m + kGrow || (m == -INFINITY && mx > -INFINITY);
      if (__any_sync(0xffffffffu, grow)) {
        const float next = grow ? mx : m;
        const float f = grow ? (m == -INFINITY ? 0.f : ex2(m - next)) : 1.f;
        if (i > 0) {
#pragma unroll 1
          for (int c = 0; c < kPD; c += 16) {
            float o[16];
            uint32_t w[16];
            tmem_ld16(t_lane + kColO + c, o);
#pragma unroll
            for (int j = 0; j < 16; ++j) w[j] = __float_as_uint(o[j] * f);
            tmem_st16(t_lane + kColO + c, w);
          }
        }
        l *= f;
        m = next;
      }
      const float ref = m == -INFINITY ? 0.f : m;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t hi[16], lw[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float x = ex2(s[half * 32 + 2 * j] - ref), y = ex2(s[half * 32 + 2 * j + 1] - ref);
          l += x + y;
          if (HALF) split_f16(x * kPScale, y * kPScale, hi[j], lw[j]);
          else split_bf16(x, y, hi[j], lw[j]);
        }
        tmem_st16(t_lane + kColHi + half * 16, hi);
        tmem_st16(t_lane + kColLo + half * 16, lw);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&s_pfull));
    }
    if (ok) ok = mbar_wait(smem_u32(&s_done), (uint32_t)(n_steps - 1) & 1u, &s_abort);
    ok = __all_sync(0xffffffffu, ok);
    if (tid == 0) pdl_trigger();
    if (ok) {
      tc_fence_after();
      const float inv = 1.f / (l * kPScale);
      T* out = (T*)a.out + (int64_t)(tile.row0 + r / R) * a.ld_out + ((int64_t)kvh * R + r % R) * kPD;
#pragma unroll 1
      for (int c = 0; c < kPD; c += 16) {
        float o[16];
        tmem_ld16(t_lane + kColO + c, o);
        uint4 w[2];
        T* t = reinterpret_cast<T*>(w);
#pragma unroll
        for (int j = 0; j < 16; ++j) t[j] = from_f32<T>(o[j] * inv);
        if (r < n_rows) {
          reinterpret_cast<uint4*>(out + c)[0] = w[0];
          reinterpret_cast<uint4*>(out + c)[1] = w[1];
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (s_abort && tid == 0 && a.err) atomicExch(a.err, HB_ERR_TIMEOUT);
  if (warp == 5)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256) : "memory");
}

// ------------------------------------------------------------------------ host
int encode_pool_map(CUtensorMap* tm, const void* pool, int64_t num_blocks, int hkv);  // attention_mma.cu

int prompt_attention_positions(const SpanAttention& a, hb_dtype dtype) {
  auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  const int R = a.kv_heads > 0 ? a.heads / a.kv_heads : 0;
  if ((dtype != HB_BF16 && dtype != HB_F16) || a.dim != kPD || a.vdim != kPD || R < 1 || R > 128 || a.gate || a.sink || a.dist_bias ||
      a.softcap > 0.f || a.key_scale || a.linear || a.tail || a.k_step.token || a.v_step.token || !(a.scale > 0.f) || a.ld_q % 8 ||
      a.ld_out % 8 || !al(a.q) || !al(a.out) || !al(a.kc) || !al(a.vc) || a.num_blocks * a.kv_heads * kBS >= (1ll << 31))
    return 0;
  return 128 / R;
}

int prompt_attention_prepare() {
  static std::mutex mu;
  static bool done[64] = {false};
  int dev = 0;
  HB_CUDA_CHECK(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  if (dev >= 0 && dev < 64 && !done[dev]) {
    HB_CUDA_CHECK(cudaFuncSetAttribute(prompt_attention_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPromptSmem));
    HB_CUDA_CHECK(cudaFuncSetAttribute(prompt_attention_kernel<__half>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPromptSmem));
    done[dev] = true;
  }
  return HB_OK;
}

int prompt_attention(cudaStream_t st, const SpanAttention& a, const RowRange* tiles, int n_tiles, hb_dtype dtype) {
  if (n_tiles == 0) return HB_OK;
  if (!prompt_attention_positions(a, dtype)) return fail(HB_ERR_INVALID_ARG, "prompt attention: sizes it does not take");
  int rc = prompt_attention_prepare();
  if (rc) return rc;
  CUtensorMap tm_k, tm_v;
  if ((rc = encode_pool_map(&tm_k, a.kc, a.num_blocks, a.kv_heads)) || (rc = encode_pool_map(&tm_v, a.vc, a.num_blocks, a.kv_heads)))
    return rc;
  const dim3 grid((unsigned)n_tiles, (unsigned)a.kv_heads);
  HB_CUDA_CHECK(launch_pdl(dtype == HB_F16 ? prompt_attention_kernel<__half> : prompt_attention_kernel<__nv_bfloat16>, grid,
                           dim3(kPromptThreads), kPromptSmem, st, tm_k, tm_v, a, tiles));
  return HB_OK;
}

}  // namespace hb
