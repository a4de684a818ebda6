// Flash attention forward on tcgen05: O = softmax(scale * Q K^T + mask) V, plus the row
// log-sum-exp needed by the backward pass.
//
// One CTA owns a tile of 128 query rows of one (batch, head); two CTAs share an SM, so that one's softmax
// runs on the CUDA cores while the tensor core works for the other, and one's start and finish hide behind
// the other's key blocks (at 512 keys a CTA has only four of them).
//
//   warp 0          TMA producer (Q once, then K and V blocks of 128 keys through rings of their own)
//   warp 1          UMMA issuer, per key block j:  O += P_{j-1} V_{j-1}  then  S = Q K_j^T
//   warps 2..5      softmax: thread r owns query row r = TMEM lane r (row max / exp2 / row sum need no shuffles)
//
// What bounds it: a TMEM round trip of a softmax warp takes hundreds of cycles behind the tensor core's own
// accumulator traffic, and eight softmax warps per SM cannot hide several of them per block; below that lies
// the exponential unit (1024 cycles per 128 x 128 block and SM).  So a thread reads its 128 scores ONCE into
// registers, P goes back into the columns of S as the TMEM operand of the second product (PV_{j-1} is issued
// before S_j, which overwrites it), and O stays in TMEM, where a warp rescales it once P_j is written (the scores'
// registers are free by then: one TMEM round trip) and only if a row maximum of its 32 rows has grown.
// P is always relative to the true running maximum, so the largest probability of a row is exactly 1 in bf16.  A
// maximum that may lag behind by 2^8 saves most of the rescaling (82.3 instead of 84.1 us at 32 x 16 heads on 512
// keys, 195 instead of 206 us at 4096 keys causal, 32 heads of 128), but then the largest probabilities are rounded
// too, and peaked rows lose precision: scores of standard deviation 3 gave 0.0021 of the output's norm off fp64
// instead of 0.0018.  Measured back to back over buffers larger than L2, two 256-row tiles' warpgroups per CTA with
// three passes over S -> now: 4096 keys causal, 32 heads of 128: 331 -> 206 us; 16 x 16 heads of 64 on 333 padded
// keys: 62 -> 36 us; 32 x 16 heads on 512 keys: 101 -> 84 us; 8 x 12 heads, 1024 keys causal, dropout: 148 -> 108 us.
//
// Replaces the eager matmul -> softmax -> dropout -> matmul attention the reference's models use
// (examples/models/gpt2/config.py:28 forces eager attention) and the SDPA/FlashAttention-2 calls
// of its sequence-parallel Llama layer (Merak/core/sequence_parallel/modeling/llama.py:24-160).
#include "attention.h"
#include "host_common.h"
#include "sm100_ptx.cuh"
#include "attention_dropout.cuh"

namespace mrk {

constexpr int kKV = 128;  // keys per block

struct AttnFwdParams {
  float* lse;                   // [B, H, Lq]
  const float* key_bias;        // optional [B, Lk], added to every score column
  int B, H, Hkv, Lq, Lk;
  int causal;
  float scale_log2;             // softmax scale * log2(e)
  float p_drop;                 // dropout on the probabilities (0 = off)
  const unsigned long long* rng;   // [seed, offset] on the device when p_drop > 0
  unsigned long long call_id;
  unsigned* status;
};

template <int D>
struct AttnFwdSmem {
  static constexpr int kTile = 128 * D * 2;                  // one Q / K / V tile
  static constexpr int kStages = (D == 64) ? 2 : 1;          // of the K ring and of the V ring
  static constexpr int kQOff = 0;
  static constexpr int kKOff = kTile;
  static constexpr int kVOff = kKOff + kStages * kTile;
  static constexpr int kBarOff = kVOff + kStages * kTile;
  static constexpr int kBiasOff = kBarOff + 256;             // 2 x 128 floats: staged key bias
  static constexpr int kTotal = kBiasOff + 1024 + 1024;      // with the alignment of the base
  static constexpr int kThreads = 192;
};

// Barrier over the 128 threads of one softmax warpgroup that also ORs a predicate (v != 0).
__device__ __forceinline__ bool named_bar_any_nonzero(uint32_t bar_id, float v) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.f32 q, %1, 0f00000000;\n\t"
      "bar.red.or.pred p, %2, 128, q;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(r) : "f"(v), "r"(bar_id) : "memory");
  return r != 0;
}

// kDrop: dropout on the probabilities.  A template argument, because a branch in the element loop cuts it into
// pieces of four exponentials whose latency nothing hides (5 % of the kernel without dropout, at 512 keys).
template <int D, bool kDrop>
__global__ void __launch_bounds__(AttnFwdSmem<D>::kThreads, 2)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                const __grid_constant__ CUtensorMap tv, const __grid_constant__ CUtensorMap to,
                const AttnFwdParams p) {
  using L = AttnFwdSmem<D>;
  constexpr int kStages = L::kStages;
  constexpr uint32_t kTmemCols = 256;      // S (then P) at column 0, O at 128
  constexpr uint32_t kOCol = 128;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBarOff);
  uint64_t* q_full = bars;                 // 1
  uint64_t* k_full = bars + 1;             // kStages each
  uint64_t* k_empty = k_full + kStages;
  uint64_t* v_full = k_empty + kStages;
  uint64_t* v_empty = v_full + kStages;
  uint64_t* s_full = v_empty + kStages;    // S_j written (and every earlier product complete)
  uint64_t* p_full = s_full + 1;           // 128 arrivals: P_j written, S_j consumed
  uint64_t* o_full = p_full + 1;           // the last P V is complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // causal: the rows with the most keys start first, so that the last CTAs to run are the short ones
  const int q_blk = p.causal ? (int)(gridDim.x - 1 - blockIdx.x) : (int)blockIdx.x;
  const int h = blockIdx.y, b = blockIdx.z;
  const int hkv = h / (p.H / p.Hkv);
  const int q0 = q_blk * 128;
  const int causal_shift = p.Lk - p.Lq;    // key j visible to query i iff j <= i + shift

  int nb = (p.Lk + kKV - 1) / kKV;         // key blocks (causal: up to the diagonal of the last row)
  if (p.causal) {
    const int last_key = min(p.Lk - 1, q0 + 127 + causal_shift);
    nb = last_key < 0 ? 0 : min(nb, last_key / kKV + 1);
  }

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    mbar_init(smem_u32(q_full), 1);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(smem_u32(&k_full[s]), 1);
      mbar_init(smem_u32(&k_empty[s]), 1);
      mbar_init(smem_u32(&v_full[s]), 1);
      mbar_init(smem_u32(&v_empty[s]), 1);
    }
    mbar_init(smem_u32(s_full), 1);
    mbar_init(smem_u32(p_full), 128);
    mbar_init(smem_u32(o_full), 1);
    fence_mbar_init();
    tma_prefetch_desc(&tq);
    tma_prefetch_desc(&tk);
    tma_prefetch_desc(&tv);
    tma_prefetch_desc(&to);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t q_smem = smem_u32(smem + L::kQOff);

  if (warp == 0) {
    if (lane == 0 && nb > 0) {
      mbar_arrive_expect_tx(smem_u32(q_full), L::kTile);
#pragma unroll
      for (int a = 0; a < D / 64; ++a)
        tma_load_4d(q_smem + a * 16384, &tq, smem_u32(q_full), a * 64, q0, h, b);
      int stage = 0;
      uint32_t phase = 0;
      for (int j = 0; j < nb; ++j) {
        if (!mbar_wait(smem_u32(&k_empty[stage]), phase ^ 1u, abort_flag, p.status)) break;
        const uint32_t kf = smem_u32(&k_full[stage]), vf = smem_u32(&v_full[stage]);
        const uint32_t ks = smem_u32(smem + L::kKOff + stage * L::kTile);
        const uint32_t vs = smem_u32(smem + L::kVOff + stage * L::kTile);
        mbar_arrive_expect_tx(kf, L::kTile);
#pragma unroll
        for (int a = 0; a < D / 64; ++a) tma_load_4d(ks + a * 16384, &tk, kf, a * 64, j * kKV, hkv, b);
        if (!mbar_wait(smem_u32(&v_empty[stage]), phase ^ 1u, abort_flag, p.status)) break;
        mbar_arrive_expect_tx(vf, L::kTile);
#pragma unroll
        for (int a = 0; a < D / 64; ++a) tma_load_4d(vs + a * 16384, &tv, vf, a * 64, j * kKV, hkv, b);
        if (++stage == kStages) { stage = 0; phase ^= 1u; }
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && nb > 0) {
      const uint32_t idesc_s = make_idesc_bf16(128, 128, 0, 0);  // Q (K-major) x K (K-major)
      const uint32_t idesc_o = make_idesc_bf16(128, D, 0, 1);    // P (TMEM) x V (MN-major)
      bool ok = mbar_wait(smem_u32(q_full), 0, abort_flag, p.status);
      int k_stage = 0, v_stage = 0;
      uint32_t k_phase = 0, v_phase = 0;
      for (int j = 0; j <= nb && ok; ++j) {
        if (j > 0) {       // softmax of block j-1 finished: P_{j-1} is ready, O is not being rescaled
          ok = mbar_wait(smem_u32(&v_full[v_stage]), v_phase, abort_flag, p.status) &&
               mbar_wait(smem_u32(p_full), (j - 1) & 1, abort_flag, p.status);
          if (!ok) break;
          tc_fence_after();
          const uint32_t vs = smem_u32(smem + L::kVOff + v_stage * L::kTile);
#pragma unroll
          for (int k = 0; k < kKV / 16; ++k)
            umma_bf16_ts(tmem_base + kOCol, tmem_base + k * 8, desc_mnmajor(vs, k, 128), idesc_o,
                         (j > 1 || k != 0) ? 1u : 0u);
          if (j < nb) umma_commit(smem_u32(&v_empty[v_stage]));
          else umma_commit(smem_u32(o_full));
          if (++v_stage == kStages) { v_stage = 0; v_phase ^= 1u; }
        }
        if (j < nb) {
          ok = mbar_wait(smem_u32(&k_full[k_stage]), k_phase, abort_flag, p.status);
          if (!ok) break;
          tc_fence_after();
          const uint32_t ks = smem_u32(smem + L::kKOff + k_stage * L::kTile);
#pragma unroll
          for (int k = 0; k < D / 16; ++k)
            umma_bf16_ss(tmem_base, desc_kmajor(q_smem + (k / 4) * 16384, k % 4),
                         desc_kmajor(ks + (k / 4) * 16384, k % 4), idesc_s, k != 0 ? 1u : 0u);
          umma_commit(smem_u32(s_full));
          umma_commit(smem_u32(&k_empty[k_stage]));
          if (++k_stage == kStages) { k_stage = 0; k_phase ^= 1u; }
        }
      }
    }
  } else {
    const int quad = warp & 3;               // TMEM lane quadrant this warp may read
    const int r = quad * 32 + lane;          // row inside the tile == TMEM lane
    const int row = q0 + r;                  // query index
    const uint32_t s_tmem = tmem_base + ((uint32_t)(quad * 32) << 16);
    const uint32_t o_tmem = s_tmem + kOCol;
    const float* kb = p.key_bias ? p.key_bias + (long long)b * p.Lk : nullptr;
    float* kbs_base = reinterpret_cast<float*>(smem + L::kBiasOff);
    float m_run = -INFINITY, l_run = 0.f;    // the maximum in use (log2 units) and the row sum relative to it
    bool ok = true;
    // dropout on the probabilities: the row sum keeps the undropped values, the P V product sees the mask
    // (the survivors' factor 1 / (1 - p) is applied to the output row)
    const uint32_t drop_thresh = attn_drop_thresh(p.p_drop);
    const uint32_t rowkey = kDrop ? attn_drop_rowkey(attn_drop_base(p.rng[0], p.rng[1] + p.call_id),
                                                    (uint32_t)(b * p.H + h), (uint32_t)row) : 0u;

    int j = 0;
    for (; j < nb && ok; ++j) {
      const int k0 = j * kKV;
      // Key bias of this block goes to shared memory once (thread r stages key k0+r, double
      // buffered); blocks whose bias is all zero (no padding) take the unbiased path.
      bool has_bias = false;
      const float* kbs = kbs_base + (j & 1) * 128;
      if (kb != nullptr) {
        const float bv = (k0 + r < p.Lk) ? __ldg(kb + k0 + r) * 1.4426950408889634f : 0.f;
        kbs_base[(j & 1) * 128 + r] = bv;
        has_bias = named_bar_any_nonzero(1, bv);
      }
      ok = mbar_wait(smem_u32(s_full), j & 1, abort_flag, p.status);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      uint32_t s[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld32(s_tmem + c * 32, s[c]);
      tmem_wait_ld();

      float sc = p.scale_log2;
      // (a negative scale turns the order of the scores round: they are scaled before the maximum is taken)
      const bool edge = (k0 + kKV > p.Lk) || (p.causal && (k0 + kKV - 1 > q0 + causal_shift)) || p.scale_log2 < 0.f;
      if (edge || has_bias) {
        const int last = p.causal ? min(p.Lk - 1, row + causal_shift) - k0 : p.Lk - 1 - k0;    // last visible column
#pragma unroll
        for (int i = 0; i < 128; i += 4) {
          const float4 bias = has_bias ? *reinterpret_cast<const float4*>(kbs + i) : make_float4(0.f, 0.f, 0.f, 0.f);
          const float bv[4] = {bias.x, bias.y, bias.z, bias.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            uint32_t& x = s[(i + e) >> 5][(i + e) & 31];
            x = __float_as_uint(i + e > last ? -INFINITY : fmaf(__uint_as_float(x), sc, bv[e]));
          }
        }
        sc = 1.f;
      }

      // ---- row maximum (in log2 units); independent partial maxima, no 128-long dependent chain ----
      float m8[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) m8[i] = __uint_as_float(s[0][i]);
#pragma unroll
      for (int i = 8; i < 128; ++i) m8[i & 7] = fmaxf(m8[i & 7], __uint_as_float(s[i >> 5][i & 31]));
      const float m_blk = fmaxf(fmaxf(fmaxf(m8[0], m8[1]), fmaxf(m8[2], m8[3])),
                                fmaxf(fmaxf(m8[4], m8[5]), fmaxf(m8[6], m8[7]))) * sc;   // a scale still to be applied is not negative
      // S_j complete means every earlier product is: nothing writes O until P_j is published
      const bool grown = j > 0 && __any_sync(0xffffffffu, m_blk > m_run);
      const float m_new = j > 0 ? fmaxf(m_run, m_blk) : m_blk;
      const float alpha = m_new == -INFINITY ? 1.f : exp2f(m_run - m_new);
      m_run = m_new;
      const float m_use = (m_run == -INFINITY) ? 0.f : m_run;

      // ---- probabilities -> TMEM (A operand of P V: two bf16 per column), row sum ----
      float l4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t packed[16];
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          float pv[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            pv[e] = exp2f(fmaf(__uint_as_float(s[c][i + e]), sc, -m_use));
            l4[e] += pv[e];
          }
          if (kDrop) {
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (!attn_drop_keep(rowkey, (uint32_t)(k0 + c * 32 + i + e), drop_thresh)) pv[e] = 0.f;
          }
          packed[i >> 1] = pack_bf16x2(pv[0], pv[1]);
          packed[(i >> 1) + 1] = pack_bf16x2(pv[2], pv[3]);
        }
        tmem_st16(s_tmem + c * 16, packed);
      }
      l_run = (grown ? l_run * alpha : l_run) + ((l4[0] + l4[1]) + (l4[2] + l4[3]));
      if (grown) {       // the scores' registers are free: one TMEM round trip for the whole row of O
        uint32_t o[D / 32][32];
#pragma unroll
        for (int c = 0; c < D / 32; ++c) tmem_ld32(o_tmem + c * 32, o[c]);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
#pragma unroll
          for (int i = 0; i < 32; ++i) o[c][i] = __float_as_uint(__uint_as_float(o[c][i]) * alpha);
          tmem_st32(o_tmem + c * 32, o[c]);
        }
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(smem_u32(p_full));
    }
    // a warp whose wait ran out still meets the others at the barriers of the blocks that they go on with
    if (!ok && kb != nullptr)
      for (++j; j < nb; ++j) named_bar_any_nonzero(1, 0.f);
    // The output leaves through the query tile's buffer (every product that reads it is complete) as a bulk
    // tensor store: a thread holds one row, so direct stores would touch 32 lines per instruction.
    // [128 q][64] bf16 boxes in the 128-byte swizzle, D / 64 of them; rows past Lq fall outside the tensor map.
    if (nb > 0 && ok) ok = mbar_wait(smem_u32(o_full), 0, abort_flag, p.status);
    ok = __all_sync(0xffffffffu, ok);
    tc_fence_after();
    const float inv = l_run > 0.f ? (kDrop ? 1.f / (1.f - p.p_drop) : 1.f) / l_run : 0.f;
    uint8_t* o_tile = smem + L::kQOff;
#pragma unroll
    for (int c = 0; c < D / 32; ++c) {
      uint32_t o[32];
      if (nb > 0 && ok) {
        tmem_ld32(o_tmem + c * 32, o);
        tmem_wait_ld();
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) o[i] = 0u;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint32_t w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
          w[e] = pack_bf16x2(__uint_as_float(o[8 * q + 2 * e]) * inv, __uint_as_float(o[8 * q + 2 * e + 1]) * inv);
        *reinterpret_cast<uint4*>(o_tile + (c >> 1) * 16384 + sw128_offset((uint32_t)r, (uint32_t)((c & 1) * 4 + q))) =
            make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
    if (row < p.Lq && p.lse)
      p.lse[((long long)b * p.H + h) * p.Lq + row] =
          l_run > 0.f ? (m_run + log2f(l_run)) * 0.6931471805599453f : -INFINITY;
    fence_proxy_async_smem();
    named_bar_sync(1, 128);
    if (r == 0 && !*abort_flag) {
#pragma unroll
      for (int a = 0; a < D / 64; ++a) tma_store_4d(&to, smem_u32(o_tile + a * 16384), a * 64, q0, h, b);
      tma_store_commit();
      tma_store_wait_read<0>();
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

template <int D, bool kDrop>
static int launch_fwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& to,
                      const AttnFwdParams& p, cudaStream_t stream) {
  using L = AttnFwdSmem<D>;
  static bool configured[64] = {false};
  int dev = 0;
  MRK_CUDA_OK(cudaGetDevice(&dev));
  if (!configured[dev & 63]) {
    MRK_CUDA_OK(cudaFuncSetAttribute(attn_fwd_kernel<D, kDrop>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kTotal));
    configured[dev & 63] = true;
  }
  dim3 grid((p.Lq + 127) / 128, p.H, p.B);
  attn_fwd_kernel<D, kDrop><<<grid, L::kThreads, L::kTotal, stream>>>(tq, tk, tv, to, p);
  MRK_CHECK_LAUNCH();
  return 0;
}

int make_bshd_tmap(CUtensorMap* out, const void* base, int D, int L, int H, int B, long long sb, long long ss,
                   long long sh, int box_rows) {
  const uint64_t dims[4] = {(uint64_t)D, (uint64_t)L, (uint64_t)H, (uint64_t)B};
  const uint64_t strides[3] = {(uint64_t)ss, (uint64_t)sh, (uint64_t)sb};
  const uint32_t box[4] = {64, (uint32_t)box_rows, 1, 1};
  return make_tmap_4d(out, base, 2, dims, strides, box, 3);
}

}  // namespace mrk

using namespace mrk;

MRK_API int mrk_attn_fwd_drop(const void* q, const void* k, const void* v, void* out, float* lse,
                              const float* key_bias, int B, int H, int Hkv, int Lq, int Lk, int D,
                              long long q_sb, long long q_ss, long long q_sh,
                              long long k_sb, long long k_ss, long long k_sh,
                              long long v_sb, long long v_ss, long long v_sh,
                              long long o_sb, long long o_ss, long long o_sh,
                              int causal, float scale, float p_drop, const void* rng, unsigned long long call_id,
                              void* stream) {
  MRK_REQUIRE(p_drop >= 0.f && p_drop < 1.f && (p_drop == 0.f || rng != nullptr), "attention: bad dropout arguments");
  MRK_REQUIRE(D == 64 || D == 128, "attention: head dim %d not supported (64 or 128)", D);
  MRK_REQUIRE(B > 0 && H > 0 && Hkv > 0 && Lq > 0 && Lk > 0 && H % Hkv == 0, "attention: bad sizes");
  MRK_REQUIRE((o_ss % 8) == 0 && (o_sh % 8) == 0 && (o_sb % 8) == 0 && ((uintptr_t)out & 15) == 0,
              "attention: output must be 16-byte aligned per row");
  CUtensorMap tq, tk, tv;
  int rc;
  if ((rc = make_bshd_tmap(&tq, q, D, Lq, H, B, q_sb, q_ss, q_sh, 128))) return rc;
  if ((rc = make_bshd_tmap(&tk, k, D, Lk, Hkv, B, k_sb, k_ss, k_sh, 128))) return rc;
  if ((rc = make_bshd_tmap(&tv, v, D, Lk, Hkv, B, v_sb, v_ss, v_sh, 128))) return rc;
  CUtensorMap to;
  if ((rc = make_bshd_tmap(&to, out, D, Lq, H, B, o_sb, o_ss, o_sh, 128))) return rc;
  AttnFwdParams p;
  p.lse = lse; p.key_bias = key_bias;
  p.B = B; p.H = H; p.Hkv = Hkv; p.Lq = Lq; p.Lk = Lk;
  p.causal = causal;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.p_drop = p_drop;
  p.rng = reinterpret_cast<const unsigned long long*>(rng);
  p.call_id = call_id;
  p.status = status_word_device();
  MRK_REQUIRE(p.status != nullptr, "attention: status word unavailable");
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (p_drop > 0.f)
    return D == 64 ? launch_fwd<64, true>(tq, tk, tv, to, p, s) : launch_fwd<128, true>(tq, tk, tv, to, p, s);
  return D == 64 ? launch_fwd<64, false>(tq, tk, tv, to, p, s) : launch_fwd<128, false>(tq, tk, tv, to, p, s);
}

MRK_API int mrk_attn_fwd(const void* q, const void* k, const void* v, void* out, float* lse,
                         const float* key_bias, int B, int H, int Hkv, int Lq, int Lk, int D,
                         long long q_sb, long long q_ss, long long q_sh,
                         long long k_sb, long long k_ss, long long k_sh,
                         long long v_sb, long long v_ss, long long v_sh,
                         long long o_sb, long long o_ss, long long o_sh,
                         int causal, float scale, void* stream) {
  return mrk_attn_fwd_drop(q, k, v, out, lse, key_bias, B, H, Hkv, Lq, Lk, D, q_sb, q_ss, q_sh, k_sb, k_ss, k_sh,
                           v_sb, v_ss, v_sh, o_sb, o_ss, o_sh, causal, scale, 0.f, nullptr, 0ull, stream);
}
