// Causal / blockwise GQA attention on tcgen05 (head dim 128 or 256), forward and backward.
//
// Forward: a CTA owns NT tiles of 128 queries of one head (NT = 1 at head dim 256, 2 at 128: with S and O of NT
// tiles tensor memory is full either way) and walks the keys in blocks of 128.
//     S  = Q K^T            tcgen05 MMA, M = 128, N = 128, K = D         -> TMEM
//     P  = exp2(S c - m)    one thread per query row (a TMEM lane is a row: no shuffles), running max m and sum l in
//                           registers; bf16 P goes back to TMEM over the columns of S it came from
//     O += P V              tcgen05 MMA, A = P from TMEM, N = D, V read MN-major from the TMA tile
// Roles: warp 0 streams K and V through a ring of five 32 KB stages, warp 1 issues the MMAs, warps 4-7 (and 8-11)
// do the softmax of tile 0 (and 1).  The tensor cores work on one S slot while the softmax works on the other: at
// NT = 1 the slots alternate by key block (S of block j + 1 is issued before O += P V of block j), at NT = 2 each
// tile has its own.  MMAs of one CTA retire in issue order, so a slot is overwritten by the next S only after its P
// has been read, without a wait.
// The accumulator O is rescaled only when a row's maximum has grown by more than 2^8 since the last rescale (the
// stale maximum keeps P <= 256, exactness is kept because l uses the same maximum).
// Query / key position offsets make the same kernel serve the hops of context-parallel ring attention: it returns the
// un-merged (O, LSE) of one key range.  Sequences of any length: rows past the end are zero-filled by TMA, masked as
// keys and clipped by the TMA store as queries.
// Bound by the tensor cores at head dim 256 and by the exponentials at 128.
// Causal, 16 x 1280 with 8 query and 2 kv heads of 256: 146 us (738 TFLOP/s), 269 us as one serial chain per CTA in
// blocks of 64 keys.  1 x 8192 of the same heads runs at 1,270 TFLOP/s, 2 x 4096 with 32 heads of 128 at 912; at 1280
// what remains is the fill and drain of each CTA's chain of 5.5 blocks on average.
// A key that a query must not see has the weight 0 in P, and 0 times a value that is not finite is NaN: such a value
// reaches every query of the tile of 128 that its key lies in, earlier ones among them.
//
// The reference calls at::scaled_dot_product_attention (src/model/qwen3_5_text.cc:1068-1075) and, for
// context parallelism, a scalar SIMT kernel (cuda/cp_attention_cuda.cu).
#include "ptx.cuh"
#include "gemm_tcgen05.h"
#include <initializer_list>
#include <type_traits>

namespace cvb {

constexpr int AT_BQ = 128;       // queries per tile
constexpr int AT_BK = 128;       // keys per block
constexpr int AT_STAGES = 5;
constexpr int AT_STAGE = 32768;  // bytes of a stage: a K or V block at head dim 128, half a block at 256

template <int D>
struct AttCfg {
  static constexpr int NT = 256 / D;                // query tiles per CTA
  static constexpr int PER = D / 128;               // stages per K or V block
  static constexpr int THREADS = 128 + 128 * NT;
  static constexpr int Q = 0;                       // NT tiles of D/64 boxes [128 x 64]
  static constexpr int RING = 65536;
  static constexpr int BARS = RING + AT_STAGES * AT_STAGE;
  static constexpr int BYTES = BARS + 256 + 1024;
};

struct AttArgs {
  float* lse;           // [B, Hq, Sq]  natural-log LSE of the scaled scores (-inf for a fully masked row)
  int Sq, Skv, Hq, Hkv, B;
  float scale_log2;     // softmax scale * log2(e)
  int causal;
  long long q_pos0, k_pos0;   // positions of query 0 and key 0 (causal: key_pos <= query_pos)
  int* status;
};

__device__ __forceinline__ uint32_t asw128(uint32_t row, uint32_t chunk) {
  return row * 128u + ((chunk ^ (row & 7u)) << 4);
}

template <int D>
__global__ void __launch_bounds__(AttCfg<D>::THREADS, 1)
attention_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                     const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO,
                     const AttArgs a) {
  using C = AttCfg<D>;
  constexpr int NT = C::NT, PER = C::PER, NB = D / 64;
  constexpr float GROW = 8.f;   // log2 of the growth that O tolerates without a rescale
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::BARS);
  uint64_t* bar_q = bars;
  uint64_t* bar_full = bars + 1;                 // [AT_STAGES]
  uint64_t* bar_empty = bar_full + AT_STAGES;    // [AT_STAGES]
  uint64_t* bar_s = bar_empty + AT_STAGES;       // [2] S of a slot is complete
  uint64_t* bar_p = bar_s + 2;                   // [2] P of a slot is in TMEM, O is rescaled
  uint64_t* bar_out = bar_p + 2;                 // [NT] the tile's output is staged
  uint64_t* bar_pen = bar_out + 2;               // NT = 1: O is complete but for the last block
  uint64_t* bar_fin = bar_pen + 1;               // every MMA is complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_fin + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // 1-D grid, last query block first: under the causal mask it sees the most keys, so the longest CTAs are
  // scheduled first and the launch ends with short ones.
  const int per_block = a.Hq * a.B;
  const int q_blocks = (a.Sq + NT * AT_BQ - 1) / (NT * AT_BQ);
  const int q0 = (q_blocks - 1 - static_cast<int>(blockIdx.x / per_block)) * (NT * AT_BQ);
  const int h = (blockIdx.x % per_block) % a.Hq;
  const int hk = h / (a.Hq / a.Hkv);
  const int b = (blockIdx.x % per_block) / a.Hq;
  const uint32_t sb = smem_u32(smem);

  // key blocks that each tile can see
  int n[NT], nmax = 0;
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    const int first = q0 + t * AT_BQ;
    int k = (a.Skv + AT_BK - 1) / AT_BK;
    if (a.causal) {
      const long long lim = a.q_pos0 + min(first + AT_BQ, a.Sq) - 1 - a.k_pos0;   // largest visible key index
      k = lim < 0 ? 0 : static_cast<int>(min(static_cast<long long>(k), lim / AT_BK + 1));
    }
    n[t] = first < a.Sq ? k : 0;
    nmax = max(nmax, n[t]);
  }

  if (tid == 0) {
    mbar_init(bar_q, 1);
    for (int s = 0; s < AT_STAGES; ++s) {
      mbar_init(&bar_full[s], 1);
      mbar_init(&bar_empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bar_s[s], 1);
      mbar_init(&bar_p[s], 4);   // one arrival per softmax warp
      mbar_init(&bar_out[s], 4);
    }
    mbar_init(bar_pen, 1);
    mbar_init(bar_fin, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  constexpr uint32_t TC_S = 0, TC_O = 256;   // S slot s at 128 s, O of tile t at 256 + t D

  auto fail = [&](int code) {
    if (!*abort_flag) atomicCAS(a.status, 0, code);
    *abort_flag = 1;
  };

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0 && nmax > 0) {
      mbar_arrive_expect_tx(bar_q, NT * D * 256);
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int c = 0; c < NB; ++c)
          tma_load_3d(smem + C::Q + (t * NB + c) * 16384, &tmQ, bar_q, h * D + c * 64, q0 + t * AT_BQ, b);
      int stage = 0;
      uint32_t phase = 0, armed = 0, parity = 0;
      bool ok = true;
      auto load = [&](int j, bool is_k) {
        for (int hf = 0; hf < PER && ok; ++hf) {
          if (!mbar_wait_bounded(&bar_empty[stage], phase ^ 1, abort_flag)) {
            fail(ERR_WAIT_EMPTY);
            ok = false;
            break;
          }
          uint8_t* dst = smem + C::RING + stage * AT_STAGE;
          mbar_arrive_expect_tx(&bar_full[stage], AT_STAGE);
          if (is_k) {   // 128 keys x 128 columns
            for (int c = 0; c < 2; ++c)
              tma_load_3d(dst + c * 16384, &tmK, &bar_full[stage], hk * D + hf * 128 + c * 64, j * AT_BK, b);
          } else {      // head dim 128: 128 keys x 128 columns; 256: 64 keys x 256 columns
            constexpr int KEYS = AT_BK / PER;
            for (int c = 0; c < NB; ++c)
              tma_load_3d(dst + c * (KEYS * 128), &tmV, &bar_full[stage], hk * D + c * 64, j * AT_BK + hf * KEYS, b);
          }
          armed |= 1u << stage;
          parity = (parity & ~(1u << stage)) | (phase << stage);
          if (++stage == AT_STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      };
      load(0, true);
      for (int j = 0; j < nmax && ok; ++j) {   // in the order in which the MMA warp takes them
        if (NT == 1) {
          if (j + 1 < nmax) load(j + 1, true);
          load(j, false);
        } else {
          load(j, false);
          if (j + 1 < nmax) load(j + 1, true);
        }
      }
      if (!ok || *abort_flag) {   // leave no copy in flight
        int dummy = 0;
        mbar_wait_bounded(bar_q, 0, &dummy);
        for (int s = 0; s < AT_STAGES; ++s)
          if (armed & (1u << s)) mbar_wait_bounded(&bar_full[s], (parity >> s) & 1, &dummy);
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer --------------------------------
    if (lane == 0 && nmax > 0) {
      constexpr uint32_t id_s = umma_idesc(128, AT_BK, 1, 0, 0);
      constexpr uint32_t id_o = umma_idesc(128, D, 1, 0, 1);
      bool ok = mbar_wait_bounded(bar_q, 0, abort_flag);
      if (!ok) fail(ERR_WAIT_FULL);
      int stage = 0;          // next stage of the ring, in the producer's order
      uint32_t phase = 0;
      auto take = [&]() {     // waits for the next stage; returns its index
        const int s = stage;
        if (ok && !mbar_wait_bounded(&bar_full[s], phase, abort_flag)) {
          fail(ERR_WAIT_FULL);
          ok = false;
        }
        if (++stage == AT_STAGES) {
          stage = 0;
          phase ^= 1;
        }
        return s;
      };
      auto qk = [&](int t, int slot, const int (&st)[2]) {
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint32_t kb = k >> 2, ks = (k & 3) * 32;
          umma_bf16(tmem_base + TC_S + slot * 128, umma_smem_desc(sb + C::Q + (t * NB + kb) * 16384 + ks, 16, 1024),
                    umma_smem_desc(sb + C::RING + st[kb >> 1] * AT_STAGE + (kb & 1) * 16384 + ks, 16, 1024), id_s,
                    k > 0);
        }
        umma_commit(&bar_s[slot]);
      };
      auto pv = [&](int t, int slot, const int (&st)[2], bool first, bool last_use) {
        tc_fence_after();
        constexpr int KEYS = AT_BK / PER;
#pragma unroll
        for (int hf = 0; hf < PER; ++hf) {
#pragma unroll
          for (int k = 0; k < KEYS / 16; ++k)
            umma_bf16_ts(tmem_base + TC_O + t * D, tmem_base + TC_S + slot * 128 + (hf * (KEYS / 16) + k) * 8,
                         umma_smem_desc(sb + C::RING + st[hf] * AT_STAGE + k * 2048, KEYS * 128, 1024), id_o,
                         !(first && hf == 0 && k == 0));
          if (last_use) umma_commit(&bar_empty[st[hf]]);
        }
      };
      auto wait_p = [&](int slot, uint32_t par) {
        if (ok && !mbar_wait_bounded(&bar_p[slot], par, abort_flag)) {
          fail(ERR_WAIT_TMEM_EMPTY);
          ok = false;
        }
      };
      int ks[2] = {0, 0}, vs[2] = {0, 0};
      for (int i = 0; i < PER; ++i) ks[i] = take();
      if (ok) {
#pragma unroll
        for (int t = 0; t < NT; ++t)
          if (n[t] > 0) qk(t, t, ks);
        for (int i = 0; i < PER; ++i) umma_commit(&bar_empty[ks[i]]);
      }
      for (int j = 0; j < nmax && ok; ++j) {
        if (NT == 1) {
          const int slot = j & 1;
          if (j + 1 < nmax) {
            for (int i = 0; i < PER; ++i) ks[i] = take();
            if (!ok) break;
            qk(0, slot ^ 1, ks);
            for (int i = 0; i < PER; ++i) umma_commit(&bar_empty[ks[i]]);
          }
          for (int i = 0; i < PER; ++i) vs[i] = take();
          wait_p(slot, (j >> 1) & 1);
          if (!ok) break;
          pv(0, slot, vs, j == 0, true);
          if (j + 2 == nmax) umma_commit(bar_pen);
        } else {
          vs[0] = take();
          if (j + 1 < nmax) ks[0] = take();
          if (!ok) break;
#pragma unroll
          for (int t = 0; t < NT; ++t) {
            if (j < n[t]) {
              wait_p(t, j & 1);
              if (!ok) break;
              pv(t, t, vs, j == 0, false);
              if (j + 1 < n[t]) qk(t, t, ks);
            }
          }
          if (!ok) break;
          umma_commit(&bar_empty[vs[0]]);
          if (j + 1 < nmax) umma_commit(&bar_empty[ks[0]]);
        }
      }
      if (ok) umma_commit(bar_fin);
    }
  } else if (warp >= 4) {
    // ------------------------------ softmax, one row per thread ---------------
    const int t = NT == 1 ? 0 : (warp >> 2) - 1;
    const int row = (warp & 3) * 32 + lane;
    const uint32_t tmem = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    const uint32_t t_o = tmem + TC_O + t * D;
    const int qi = q0 + t * AT_BQ + row;
    const long long qpos = a.q_pos0 + qi;
    const long long first_pos = a.q_pos0 + q0 + t * AT_BQ;
    const int nt = t == 0 ? n[0] : n[NT - 1];
    float m_used = -INFINITY, l = 0.f;   // the maximum that O and l refer to; sum of the weights
    bool ok = true;
    auto wait = [&](uint64_t* bar, uint32_t par) {
      ok = __all_sync(0xffffffffu, mbar_wait_bounded(bar, par, abort_flag));
      if (!ok && lane == 0) fail(ERR_WAIT_TMEM_FULL);
      return ok;
    };
    for (int j = 0; j < nt; ++j) {
      const int slot = NT == 1 ? (j & 1) : t;
      if (!wait(&bar_s[slot], NT == 1 ? (j >> 1) & 1 : j & 1)) break;
      tc_fence_after();
      const uint32_t t_s = tmem + TC_S + slot * 128;
      uint32_t r[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32(t_s + c * 32, r[c]);
      tmem_ld_wait();
      const int k0 = j * AT_BK;
      // only the blocks on the diagonal and the last one hold keys that some row must not see
      if (k0 + AT_BK > a.Skv || (a.causal && a.k_pos0 + k0 + AT_BK - 1 > first_pos)) {
        long long vis64 = a.Skv - k0;
        if (a.causal) vis64 = min(vis64, qpos - (a.k_pos0 + k0) + 1);
        const int vis = static_cast<int>(max(min(vis64, static_cast<long long>(AT_BK)), 0ll));
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c * 32 + i >= vis) r[c][i] = __float_as_uint(-INFINITY);
      }
      float mx[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        mx[c] = __uint_as_float(r[c][0]);
#pragma unroll
        for (int i = 1; i < 32; ++i) mx[c] = fmaxf(mx[c], __uint_as_float(r[c][i]));
      }
      const float m_blk = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * a.scale_log2;   // scale > 0
      const bool want = (m_blk > m_used + GROW) || (m_used == -INFINITY && m_blk > -INFINITY);
      const bool grow = __any_sync(0xffffffffu, want);   // warp-uniform: tcgen05.ld / st are warp-collective
      float alpha = 1.f;
      if (grow) {
        const float m_new = fmaxf(m_used, m_blk);
        alpha = m_used == -INFINITY ? 0.f : exp2f(m_used - m_new);
        m_used = m_new;
        l *= alpha;
      }
      const float mm = m_used == -INFINITY ? 0.f : m_used;
      float sum[4];
      uint32_t p[4][16];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        sum[c] = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float p0 = exp2f(__uint_as_float(r[c][2 * i]) * a.scale_log2 - mm);
          const float p1 = exp2f(__uint_as_float(r[c][2 * i + 1]) * a.scale_log2 - mm);
          sum[c] += p0 + p1;
          p[c][i] = pack_bf16x2(p0, p1);
        }
      }
      l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
      if (grow && j > 0) {
        // O must hold the blocks before.  At NT = 2 that is so once S of this block is complete, at NT = 1 once S of
        // the next one is (both were issued after O += P V of block j - 1, and a commit covers all MMAs issued before
        // it); before the last block there is a barrier of its own.
        if (NT == 1) {
          if (j + 1 < nt ? !wait(&bar_s[slot ^ 1], ((j + 1) >> 1) & 1) : !wait(bar_pen, 0)) break;
          tc_fence_after();
        }
#pragma unroll 1
        for (int c0 = 0; c0 < D; c0 += 16) {
          uint32_t o[16];
          tmem_ld_32x16(t_o + c0, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          tmem_st_32x16(t_o + c0, o);
        }
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_st_32x16(t_s + c * 16, p[c]);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_p[slot]);
    }
    // a CTA without visible keys has loaded nothing; otherwise every MMA is over, and with them every load
    if (ok && nmax > 0) wait(bar_fin, 0);
    if (ok && q0 + t * AT_BQ < a.Sq) {
      tc_fence_after();
      // O / l as bf16 over this tile's Q (its last S is complete), then out by TMA, which drops rows past the end
      const float inv = l > 0.f ? 1.f / l : 0.f;
      uint8_t* stage = smem + C::Q + t * (D * 256);
#pragma unroll 1
      for (int c0 = 0; c0 < D; c0 += 32) {
        uint32_t o[32];
        if (nt > 0) {
          tmem_ld_32x32(t_o + c0, o);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = 0u;
        }
        uint8_t* box = stage + (c0 >> 6) * 16384;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint4 u;
          u.x = pack_bf16x2(__uint_as_float(o[8 * c + 0]) * inv, __uint_as_float(o[8 * c + 1]) * inv);
          u.y = pack_bf16x2(__uint_as_float(o[8 * c + 2]) * inv, __uint_as_float(o[8 * c + 3]) * inv);
          u.z = pack_bf16x2(__uint_as_float(o[8 * c + 4]) * inv, __uint_as_float(o[8 * c + 5]) * inv);
          u.w = pack_bf16x2(__uint_as_float(o[8 * c + 6]) * inv, __uint_as_float(o[8 * c + 7]) * inv);
          *reinterpret_cast<uint4*>(box + asw128(row, ((c0 & 32) >> 3) + c)) = u;
        }
      }
      if (qi < a.Sq)
        a.lse[(static_cast<long long>(b) * a.Hq + h) * a.Sq + qi] =
            l > 0.f ? (m_used + log2f(l)) * 0.6931471805599453f : -INFINITY;
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_out[t]);
      if (row == 0 && mbar_wait_bounded(&bar_out[t], 0, abort_flag)) {
#pragma unroll
        for (int c = 0; c < NB; ++c)
          tma_store_3d(&tmO, stage + c * 16384, h * D + c * 64, q0 + t * AT_BQ, b);
        tma_store_commit();
        tma_store_wait_read();
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <int D>
static int launch_fwd(const void* q, const void* k, const void* v, void* out, float* lse, long long B, int Sq,
                      int Skv, int Hq, int Hkv, float scale, int causal, long long q_pos0, long long k_pos0,
                      int* status, cudaStream_t st) {
  using C = AttCfg<D>;
  CUtensorMap mq, mk, mv, mo;
  const uint64_t qc = static_cast<uint64_t>(Hq) * D, kc = static_cast<uint64_t>(Hkv) * D;
  if (make_tensor_map_3d(&mq, q, 2, qc, Sq, B, qc * 2, qc * 2 * Sq, 64, AT_BQ) ||
      make_tensor_map_3d(&mo, out, 2, qc, Sq, B, qc * 2, qc * 2 * Sq, 64, AT_BQ) ||
      make_tensor_map_3d(&mk, k, 2, kc, Skv, B, kc * 2, kc * 2 * Skv, 64, AT_BK) ||
      make_tensor_map_3d(&mv, v, 2, kc, Skv, B, kc * 2, kc * 2 * Skv, 64, AT_BK / C::PER))
    return -10;
  AttArgs a{};
  a.lse = lse; a.Sq = Sq; a.Skv = Skv; a.Hq = Hq; a.Hkv = Hkv;
  a.B = static_cast<int>(B);
  a.scale_log2 = scale * 1.4426950408889634f; a.causal = causal; a.q_pos0 = q_pos0; a.k_pos0 = k_pos0;
  a.status = status;
  static bool attr = false;
  if (!attr) {
    if (cudaFuncSetAttribute(attention_fwd_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::BYTES) !=
        cudaSuccess)
      return -11;
    attr = true;
  }
  const long long blocks = static_cast<long long>((Sq + C::NT * AT_BQ - 1) / (C::NT * AT_BQ)) * Hq * B;
  if (blocks > 0x7fffffffLL) return -2;
  attention_fwd_kernel<D><<<static_cast<unsigned>(blocks), C::THREADS, C::BYTES, st>>>(mq, mk, mv, mo, a);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace cvb

using namespace cvb;

// q: bf16 [B, Sq, Hq, D]; k, v: bf16 [B, Skv, Hkv, D] (all contiguous); out: bf16 [B, Sq, Hq, D];
// lse: fp32 [B, Hq, Sq].  D in {128, 256}; Hq % Hkv == 0; any Sq and Skv.
// causal != 0 masks keys whose position (k_pos0 + index) exceeds the query's (q_pos0 + index).
extern "C" int cvb_attention_fwd(const void* q, const void* k, const void* v, void* out, float* lse, long long B,
                                 int Sq, int Skv, int Hq, int Hkv, int D, float scale, int causal, long long q_pos0,
                                 long long k_pos0, int* status, void* stream) {
  if (B <= 0 || Sq <= 0 || Skv <= 0) return 0;
  if (Hkv <= 0 || Hq % Hkv || !(scale > 0.f)) return -1;
  if (B * Sq > 0x7fffffffLL || B * Skv > 0x7fffffffLL) return -2;
  for (const void* p : {q, k, v, static_cast<const void*>(out)})
    if (reinterpret_cast<uintptr_t>(p) & 15) return -3;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (D != 128 && D != 256) return -1;
  auto launch = D == 128 ? launch_fwd<128> : launch_fwd<256>;
  return launch(q, k, v, out, lse, B, Sq, Skv, Hq, Hkv, scale, causal, q_pos0, k_pos0, status, st);
}

// =================================================================================================
// Backward.
//
// One kernel template in four roles, each with an accumulator that stays in TMEM for the whole CTA:
//   BWD_Q   rows = 128 queries, walks the keys:     dQ += dS K
//   BWD_K   rows = 128 keys, walks the queries:     dK += dS^T Q                    (head dim 256)
//   BWD_V   rows = 128 keys, walks the queries:     dV += P^T dO                    (head dim 256)
//   BWD_KV  both of the last two in one CTA                                         (head dim 128)
// At head dim 256 the accumulators of dK and dV alone fill the 512 TMEM columns, so the two are separate launches.
// The walk goes in steps of 64 columns (queries or keys).  With A1, A2 the CTA's own rows (K and V, or Q and dO) and
// B1, B2 the step's rows of the other side (Q and dO, or K and V):
//     S  = A1 B1^T       dP = A2 B2^T           M = 128, N = 64, K = D
//     P  = exp2(S c - LSE)          dS = P (dP - Delta) scale
//     acc += dS B1  (and acc_v += P B2)         M = 128, N = D, K = 64, B read MN-major
// dQ needs no reduction across CTAs (no zeroed fp32 buffer, no transposing pass over it) at the price of forming S and
// dP once more.
// What makes the pipeline fit into 227 KB at head dim 256: A2 is copied once into 128 TMEM columns and read from there
// as the A operand, which leaves three slots for the operand that is held until its accumulate step and one for the
// other; S and dP have one TMEM buffer each, which the softmax warps empty into registers and release at once.  The
// tensor cores then run S, dP of step j + 1 while the warps form dS of step j, and the accumulate step of j while
// the warps fetch S, dP of j + 1.
// Roles: warp 0 TMA producer, warp 1 MMA issuer, warps 2-9 two warpgroups that split the 64 columns of a step.
// A CTA of BWD_K / BWD_V / BWD_KV walks the queries of EVERY head of its GQA group, so dK / dV come out summed.
// Causal, 16 x 1280 with 8 query and 2 kv heads of 256: dQ 232, dK 209, dV 145 and Delta 31 us; one serial chain of MMA
// and softmax per CTA in two kernels, with dQ reduced into a cleared fp32 buffer and transposed, took 1,130.  A step of
// 64 columns of BWD_K takes about 1.9 us: three MMA units against 64 KB of operands, as many bytes per unit as the
// forward reads.
// =================================================================================================
constexpr int AB_ROWS = 128;   // rows per CTA
constexpr int AB_STEP = 64;    // columns per step
constexpr int AB_THREADS = 320;

enum : int { BWD_Q = 0, BWD_K = 1, BWD_V = 2, BWD_KV = 3 };

template <int D, int MODE>
struct AttBwdCfg {
  static constexpr bool ROWQ = MODE == BWD_Q;              // rows are queries
  static constexpr bool HAS_DP = MODE != BWD_V;
  static constexpr bool ACC_1 = MODE != BWD_V;             // acc += dS B1
  static constexpr bool ACC_V = MODE == BWD_V || MODE == BWD_KV;
  static constexpr int BLOCK = D * 128;                    // bytes of one [64 x D] block
  // ring 1 holds B1, ring 2 holds B2.  An operand that an accumulate step reads is held for a whole step longer than
  // one that only S or dP reads; BWD_V takes them in different MMAs and balances the two.
  static constexpr int N1 = MODE == BWD_V ? 2 : 3;
  static constexpr int N2 = MODE == BWD_V ? 2 : (MODE == BWD_KV ? 3 : (D == 128 ? 2 : 1));
  static constexpr int A1 = 0;                             // D/64 boxes [128 x 64]
  static constexpr int R1 = A1 + D * 256;
  static constexpr int R2 = R1 + N1 * BLOCK;
  static constexpr int PT = R2 + N2 * BLOCK;               // P   [128 x 64] bf16
  static constexpr int DS = PT + (ACC_V ? 16384 : 0);      // dS  [128 x 64] bf16
  static constexpr int VEC = DS + (ACC_1 ? 16384 : 0);     // per warp: lse2[32], delta[32]
  static constexpr int BARS = VEC + 2048;
  static constexpr int BYTES = BARS + 256 + 1024;
  static constexpr int STG_A2 = R1 + BLOCK;                // A2 on its way to TMEM: slots 1 and 2 of ring 1
  static constexpr int STG_V = (MODE == BWD_KV) ? R2 : A1; // dV on its way out
  static constexpr uint32_t TC_1 = 0, TC_V = (MODE == BWD_KV) ? D : 0, TC_A2 = 256, TC_S = 384, TC_DP = 448;
};

struct AttBwdArgs {
  const float* lse;      // [B, Hq, Sq] natural log
  const float* delta;    // [B, Hq, Sq] rowsum(dO * O)
  int Sq, Skv, Hq, Hkv, B;
  float scale, scale_log2;
  int causal;
  long long q_pos0, k_pos0;
  int* status;
};

// Maps: tmA1 / tmA2 boxes of 128 rows, tmB1 / tmB2 boxes of 64 rows, tmO1 (dQ or dK) / tmOV (dV) boxes of 128 rows.
template <int D, int MODE>
__global__ void __launch_bounds__(AB_THREADS, 1)
attention_bwd_kernel(const __grid_constant__ CUtensorMap tmA1, const __grid_constant__ CUtensorMap tmA2,
                     const __grid_constant__ CUtensorMap tmB1, const __grid_constant__ CUtensorMap tmB2,
                     const __grid_constant__ CUtensorMap tmO1, const __grid_constant__ CUtensorMap tmOV,
                     const AttBwdArgs a) {
  using C = AttBwdCfg<D, MODE>;
  constexpr int NB = D / 64;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::BARS);
  uint64_t* bar_a = bars;            // A1 has landed
  uint64_t* bar_a2 = bars + 1;       // A2 is in TMEM
  uint64_t* bar_sd = bars + 2;       // S and dP of a step are complete
  uint64_t* bar_free = bars + 3;     // S and dP have been read
  uint64_t* bar_ds = bars + 4;       // P / dS of a step are in shared memory
  uint64_t* bar_acc = bars + 5;      // the accumulate step is complete
  uint64_t* full1 = bars + 6;        // [3]
  uint64_t* empty1 = bars + 9;       // [3]
  uint64_t* full2 = bars + 12;       // [3]
  uint64_t* empty2 = bars + 15;      // [3]
  uint64_t* bar_out = bars + 18;     // the result is staged
  uint64_t* bar_a2s = bars + 19;     // A2 has landed in its staging slots
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 20);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t sb = smem_u32(smem);
  const int group = a.Hq / a.Hkv;   // query heads that share a kv head
  // 1-D grid, row block slowest and the longest first: under the causal mask late queries see the most keys and
  // early keys are seen by the most queries.
  const int heads = C::ROWQ ? a.Hq : a.Hkv;
  const int per_block = heads * a.B;
  const int row_blocks = ((C::ROWQ ? a.Sq : a.Skv) + AB_ROWS - 1) / AB_ROWS;
  const int blk = static_cast<int>(blockIdx.x) / per_block;
  const int r0 = (C::ROWQ ? row_blocks - 1 - blk : blk) * AB_ROWS;
  const int head = static_cast<int>(blockIdx.x % per_block) % heads;
  const int b = static_cast<int>(blockIdx.x % per_block) / heads;
  const int hq0 = C::ROWQ ? head : head * group;
  const int hk = C::ROWQ ? head / group : head;

  // steps: column blocks [c_begin, c_end) for each query head of the group
  int c_begin = 0, c_end = ((C::ROWQ ? a.Skv : a.Sq) + AB_STEP - 1) / AB_STEP;
  if (a.causal) {
    if (C::ROWQ) {   // keys up to the last query of the block
      const long long lim = a.q_pos0 + min(r0 + AB_ROWS, a.Sq) - 1 - a.k_pos0;
      c_end = lim < 0 ? 0 : static_cast<int>(min(static_cast<long long>(c_end), lim / AB_STEP + 1));
    } else {         // queries from the first key of the block on
      const long long need = a.k_pos0 + r0 - a.q_pos0 - (AB_STEP - 1);
      if (need > 0) c_begin = static_cast<int>(min(static_cast<long long>(c_end), (need + AB_STEP - 1) / AB_STEP));
    }
  }
  const int per_head = c_end - c_begin;
  const int steps = per_head * (C::ROWQ ? 1 : group);

  if (tid == 0) {
    mbar_init(bar_a, 1);
    mbar_init(bar_a2, 8);
    mbar_init(bar_a2s, 1);
    mbar_init(bar_sd, 1);
    mbar_init(bar_free, 8);
    mbar_init(bar_ds, 8);
    mbar_init(bar_acc, 1);
    mbar_init(bar_out, 8);
    for (int s = 0; s < 3; ++s) {
      mbar_init(&full1[s], 1);
      mbar_init(&empty1[s], 1);
      mbar_init(&full2[s], 1);
      mbar_init(&empty2[s], 1);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmA1);
    tma_prefetch_desc(&tmB1);
    tma_prefetch_desc(&tmB2);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  auto fail = [&](int code) {
    if (!*abort_flag) atomicCAS(a.status, 0, code);
    *abort_flag = 1;
  };

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0 && steps > 0) {
      const int ha = C::ROWQ ? head : hk;
      mbar_arrive_expect_tx(bar_a, D * 256u);
#pragma unroll
      for (int c = 0; c < NB; ++c) tma_load_3d(smem + C::A1 + c * 16384, &tmA1, bar_a, ha * D + c * 64, r0, b);
      bool ok = true;
      uint32_t armed = 0, parity = 0;
      // slot and phase of step j in a ring of n slots
      auto load = [&](int j, int ring) {
        const int n = ring == 1 ? C::N1 : C::N2;
        const int slot = j % n;
        const uint32_t ph = (j / n) & 1;
        uint64_t* fb = (ring == 1 ? full1 : full2) + slot;
        if (!mbar_wait_bounded((ring == 1 ? empty1 : empty2) + slot, ph ^ 1, abort_flag)) {
          fail(ERR_WAIT_EMPTY);
          ok = false;
          return;
        }
        const int col = (c_begin + j % per_head) * AB_STEP;
        const int hb = C::ROWQ ? hk : hq0 + j / per_head;
        uint8_t* dst = smem + (ring == 1 ? C::R1 : C::R2) + slot * C::BLOCK;
        mbar_arrive_expect_tx(fb, C::BLOCK);
#pragma unroll
        for (int c = 0; c < NB; ++c)
          tma_load_3d(dst + c * 8192, ring == 1 ? &tmB1 : &tmB2, fb, hb * D + c * 64, col, b);
        const int bit = (ring == 1 ? 0 : 3) + slot;
        armed |= 1u << bit;
        parity = (parity & ~(1u << bit)) | (ph << bit);
      };
      load(0, 1);     // S of step 0 starts while A2 is on its way
      if (C::HAS_DP) {
        mbar_arrive_expect_tx(bar_a2s, D * 256u);
#pragma unroll
        for (int c = 0; c < NB; ++c) tma_load_3d(smem + C::STG_A2 + c * 16384, &tmA2, bar_a2s, ha * D + c * 64, r0, b);
      }
      if (ok) load(0, 2);
      if (ok && C::HAS_DP && !mbar_wait_bounded(bar_a2, 0, abort_flag)) {   // slots 1 and 2 of ring 1 held A2
        fail(ERR_WAIT_EMPTY);
        ok = false;
      }
      for (int j = 1; j < steps && ok; ++j) {
        load(j, 1);
        if (ok) load(j, 2);
      }
      if (!ok || *abort_flag) {   // leave no copy in flight
        int dummy = 0;
        mbar_wait_bounded(bar_a, 0, &dummy);
        if (C::HAS_DP) mbar_wait_bounded(bar_a2s, 0, &dummy);
        for (int s = 0; s < 6; ++s)
          if (armed & (1u << s)) mbar_wait_bounded((s < 3 ? full1 + s : full2 + s - 3), (parity >> s) & 1, &dummy);
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer --------------------------------
    if (lane == 0 && steps > 0) {
      constexpr uint32_t id_s = umma_idesc(128, AB_STEP, 1, 0, 0);
      constexpr uint32_t id_acc = umma_idesc(128, D, 1, 0, 1);
      bool ok = true;
      auto wait = [&](uint64_t* bar, uint32_t par, int code) {
        if (ok && !mbar_wait_bounded(bar, par, abort_flag)) {
          fail(code);
          ok = false;
        }
      };
      auto scores = [&](int j) {   // S (and dP) of step j
        const int s1 = j % C::N1, s2 = j % C::N2;
        wait(&full1[s1], (j / C::N1) & 1, ERR_WAIT_FULL);
        if (!ok) return;
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint32_t kb = k >> 2, ks = (k & 3) * 32;
          umma_bf16(tmem_base + C::TC_S, umma_smem_desc(sb + C::A1 + kb * 16384 + ks, 16, 1024),
                    umma_smem_desc(sb + C::R1 + s1 * C::BLOCK + kb * 8192 + ks, 16, 1024), id_s, k > 0);
        }
        if (!C::ACC_1) umma_commit(&empty1[s1]);
        if (C::HAS_DP) {
          if (j == 0) wait(bar_a2, 0, ERR_WAIT_FULL);
          wait(&full2[s2], (j / C::N2) & 1, ERR_WAIT_FULL);
          if (!ok) return;
          tc_fence_after();
#pragma unroll
          for (int k = 0; k < D / 16; ++k) {
            const uint32_t kb = k >> 2, ks = (k & 3) * 32;
            umma_bf16_ts(tmem_base + C::TC_DP, tmem_base + C::TC_A2 + k * 8,
                         umma_smem_desc(sb + C::R2 + s2 * C::BLOCK + kb * 8192 + ks, 16, 1024), id_s, k > 0);
          }
          if (!C::ACC_V) umma_commit(&empty2[s2]);
        }
        umma_commit(bar_sd);
      };
      wait(bar_a, 0, ERR_WAIT_FULL);
      if (ok) scores(0);
      for (int j = 0; j < steps && ok; ++j) {
        if (j + 1 < steps) {
          wait(bar_free, j & 1, ERR_WAIT_TMEM_EMPTY);
          if (!ok) break;
          scores(j + 1);
          if (!ok) break;
        }
        const int s1 = j % C::N1, s2 = j % C::N2;
        wait(bar_ds, j & 1, ERR_WAIT_TMEM_EMPTY);
        if (C::ACC_V && !C::HAS_DP) wait(&full2[s2], (j / C::N2) & 1, ERR_WAIT_FULL);
        if (!ok) break;
        tc_fence_after();
        if (C::ACC_V) {
#pragma unroll
          for (int k = 0; k < AB_STEP / 16; ++k)
            umma_bf16(tmem_base + C::TC_V, umma_smem_desc(sb + C::PT + k * 32, 16, 1024),
                      umma_smem_desc(sb + C::R2 + s2 * C::BLOCK + k * 2048, 8192, 1024), id_acc, (j > 0 || k > 0));
          umma_commit(&empty2[s2]);
        }
        if (C::ACC_1) {
#pragma unroll
          for (int k = 0; k < AB_STEP / 16; ++k)
            umma_bf16(tmem_base + C::TC_1, umma_smem_desc(sb + C::DS + k * 32, 16, 1024),
                      umma_smem_desc(sb + C::R1 + s1 * C::BLOCK + k * 2048, 8192, 1024), id_acc, (j > 0 || k > 0));
          umma_commit(&empty1[s1]);
        }
        umma_commit(bar_acc);
      }
    }
  } else {
    // ------------------------------ P and dS, one row per thread and half ---------------
    const int wg = warp >= 6 ? 1 : 0;       // columns [32 wg, 32 wg + 32) of every step
    const int quad = warp & 3;              // TMEM lane quadrant of this warp
    const int row = quad * 32 + lane;
    float* v_lse2 = reinterpret_cast<float*>(smem + C::VEC) + (warp - 2) * 64;
    float* v_delta = v_lse2 + 32;
    const uint32_t tmem = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    const int ri = r0 + row;
    bool ok = true;
    auto wait = [&](uint64_t* bar, uint32_t par) {
      ok = __all_sync(0xffffffffu, mbar_wait_bounded(bar, par, abort_flag));
      if (!ok && lane == 0) fail(ERR_WAIT_TMEM_FULL);
      return ok;
    };
    // queries past the end, and queries that see no key, get LSE = +inf: their P is exp2(-inf) = 0
    auto lse2_of = [](float lse) { return lse > -INFINITY ? lse * 1.4426950408889634f : INFINITY; };
    float row_lse2 = INFINITY, row_delta = 0.f;
    if (C::ROWQ && ri < a.Sq) {
      const long long i = (static_cast<long long>(b) * a.Hq + head) * a.Sq + ri;
      row_lse2 = lse2_of(a.lse[i]);
      row_delta = a.delta[i];
    }
    if (C::HAS_DP && steps > 0 && wait(bar_a2s, 0)) {
      // this row's A2 into TMEM, two bf16 per column: the A operand of dP
#pragma unroll 1
      for (int c = wg * (NB / 2); c < (wg + 1) * (NB / 2); ++c) {
        uint32_t r[32];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint4 u = *reinterpret_cast<const uint4*>(smem + C::STG_A2 + c * 16384 + asw128(row, i));
          r[4 * i] = u.x;
          r[4 * i + 1] = u.y;
          r[4 * i + 2] = u.z;
          r[4 * i + 3] = u.w;
        }
        tmem_st_32x32(tmem + C::TC_A2 + c * 32, r);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_a2);
    }
    const long long row_pos = (C::ROWQ ? a.q_pos0 : a.k_pos0) + ri;
    for (int j = 0; j < steps && ok; ++j) {
      const int col0 = (c_begin + j % per_head) * AB_STEP + wg * 32;   // first column of this thread's half
      if (!C::ROWQ) {   // the scalars of this half's queries, one copy per warp: no barrier between warps
        const int qi = col0 + lane;
        const long long i = (static_cast<long long>(b) * a.Hq + hq0 + j / per_head) * a.Sq + qi;
        const float l2 = qi < a.Sq ? lse2_of(a.lse[i]) : INFINITY;
        const float dl = C::HAS_DP && qi < a.Sq ? a.delta[i] : 0.f;
        __syncwarp();
        v_lse2[lane] = l2;
        v_delta[lane] = dl;
        __syncwarp();
      }
      if (!wait(bar_sd, j & 1)) break;
      tc_fence_after();
      uint32_t rs[32], rp[32];
      tmem_ld_32x32(tmem + C::TC_S + wg * 32, rs);
      if (C::HAS_DP) tmem_ld_32x32(tmem + C::TC_DP + wg * 32, rp);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_free);
      uint32_t pk[16], dk[16];
      auto form = [&](auto masked, int lo, int hi) {
        constexpr bool MASKED = decltype(masked)::value;
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          float4 l2, dl;
          if (C::ROWQ) {
            l2 = make_float4(row_lse2, row_lse2, row_lse2, row_lse2);
            dl = make_float4(row_delta, row_delta, row_delta, row_delta);
          } else {
            l2 = *reinterpret_cast<const float4*>(v_lse2 + i);
            if (C::HAS_DP) dl = *reinterpret_cast<const float4*>(v_delta + i);
          }
          const float l2v[4] = {l2.x, l2.y, l2.z, l2.w}, dlv[4] = {dl.x, dl.y, dl.z, dl.w};
          float p[4], ds[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            p[e] = exp2f(__uint_as_float(rs[i + e]) * a.scale_log2 - l2v[e]);
            if (MASKED && (i + e < lo || i + e >= hi)) p[e] = 0.f;
            if (C::HAS_DP) ds[e] = p[e] * (__uint_as_float(rp[i + e]) - dlv[e]) * a.scale;
          }
#pragma unroll
          for (int e = 0; e < 4; e += 2) {
            if (C::ACC_V) pk[(i + e) / 2] = pack_bf16x2(p[e], p[e + 1]);
            if (C::ACC_1) dk[(i + e) / 2] = pack_bf16x2(ds[e], ds[e + 1]);
          }
        }
      };
      // columns [lo, hi) of this half are visible from this row; most steps are visible from every row of the warp
      int lo = 0, hi = 32;
      if (C::ROWQ) {
        long long v = a.Skv - col0;
        if (a.causal) v = min(v, row_pos - (a.k_pos0 + col0) + 1);
        hi = static_cast<int>(max(min(v, 32ll), 0ll));
      } else if (a.causal) {
        lo = static_cast<int>(max(min(row_pos - (a.q_pos0 + col0), 32ll), 0ll));
      }
      if (__any_sync(0xffffffffu, lo > 0 || hi < 32)) form(std::true_type{}, lo, hi);
      else form(std::false_type{}, lo, hi);
      if (j > 0 && !wait(bar_acc, (j - 1) & 1)) break;   // the previous step has read the buffers
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const uint32_t off = asw128(row, wg * 4 + c);
        if (C::ACC_V)
          *reinterpret_cast<uint4*>(smem + C::PT + off) =
              make_uint4(pk[4 * c], pk[4 * c + 1], pk[4 * c + 2], pk[4 * c + 3]);
        if (C::ACC_1)
          *reinterpret_cast<uint4*>(smem + C::DS + off) =
              make_uint4(dk[4 * c], dk[4 * c + 1], dk[4 * c + 2], dk[4 * c + 3]);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_ds);
    }
    if (ok && steps > 0) wait(bar_acc, (steps - 1) & 1);
    if (ok) {
      tc_fence_after();
      // accumulators as bf16 over operands that are no longer read, then out by TMA, which drops rows past the end
#pragma unroll
      for (int which = 0; which < 2; ++which) {
        if ((which == 0 && !C::ACC_1) || (which == 1 && !C::ACC_V)) continue;
        uint8_t* stage = smem + (which == 0 ? C::A1 : C::STG_V);
        const uint32_t tc = which == 0 ? C::TC_1 : C::TC_V;
#pragma unroll 1
        for (int c0 = wg * 32; c0 < D; c0 += 64) {
          uint32_t o[32];
          if (steps > 0) {
            tmem_ld_32x32(tmem + tc + c0, o);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = 0u;
          }
          uint8_t* box = stage + (c0 >> 6) * 16384;
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint4 u;
            u.x = pack_bf16x2(__uint_as_float(o[8 * c + 0]), __uint_as_float(o[8 * c + 1]));
            u.y = pack_bf16x2(__uint_as_float(o[8 * c + 2]), __uint_as_float(o[8 * c + 3]));
            u.z = pack_bf16x2(__uint_as_float(o[8 * c + 4]), __uint_as_float(o[8 * c + 5]));
            u.w = pack_bf16x2(__uint_as_float(o[8 * c + 6]), __uint_as_float(o[8 * c + 7]));
            *reinterpret_cast<uint4*>(box + asw128(row, wg * 4 + c)) = u;
          }
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_out);
      if (tid == 64 && mbar_wait_bounded(bar_out, 0, abort_flag)) {
#pragma unroll
        for (int c = 0; c < NB; ++c) {
          if (C::ACC_1) tma_store_3d(&tmO1, smem + C::A1 + c * 16384, head * D + c * 64, r0, b);
          if (C::ACC_V) tma_store_3d(&tmOV, smem + C::STG_V + c * 16384, head * D + c * 64, r0, b);
        }
        tma_store_commit();
        tma_store_wait_read();
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// delta[b, h, q] = sum_d dO[b, q, h, d] * O[b, q, h, d]     (a warp takes DELTA_ROWS (token, head) rows of up to 256)
// HBM-bound; with one row per warp the index arithmetic of the store was as long as the row (16 x 1280 x 8 of 256:
// 37 -> 31 us)
constexpr int DELTA_ROWS = 4;
__global__ void __launch_bounds__(256)
attention_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o,
                       float* __restrict__ delta, long long rows, int Sq, int Hq, int D) {
  // rows are (b * Sq + q) * Hq + h
  const long long row0 = ((static_cast<long long>(blockIdx.x) * 256 + threadIdx.x) >> 5) * DELTA_ROWS;
  const int lane = threadIdx.x & 31;
  const int c = lane * 8;
  uint4 a[DELTA_ROWS], g[DELTA_ROWS];
#pragma unroll
  for (int u = 0; u < DELTA_ROWS; ++u) {
    const bool ok = row0 + u < rows && c < D;
    a[u] = ok ? *reinterpret_cast<const uint4*>(o + (row0 + u) * D + c) : make_uint4(0u, 0u, 0u, 0u);
    g[u] = ok ? *reinterpret_cast<const uint4*>(d_o + (row0 + u) * D + c) : make_uint4(0u, 0u, 0u, 0u);
  }
  float mine = 0.f;
#pragma unroll
  for (int u = 0; u < DELTA_ROWS; ++u) {
    const __nv_bfloat162* pa = reinterpret_cast<const __nv_bfloat162*>(&a[u]);
    const __nv_bfloat162* pg = reinterpret_cast<const __nv_bfloat162*>(&g[u]);
    float acc = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 x = __bfloat1622float2(pa[j]), y = __bfloat1622float2(pg[j]);
      acc += x.x * y.x + x.y * y.y;
    }
    acc = warp_sum(acc);
    if (lane == u) mine = acc;
  }
  const long long row = row0 + lane;
  if (lane < DELTA_ROWS && row < rows) {
    const long long bq = row / Hq, h = row - bq * Hq, b = bq / Sq, q = bq - b * Sq;
    delta[(b * Hq + h) * Sq + q] = mine;
  }
}

template <int D, int MODE>
static int launch_bwd(const CUtensorMap& a1, const CUtensorMap& a2, const CUtensorMap& b1, const CUtensorMap& b2,
                      const CUtensorMap& o1, const CUtensorMap& ov, const AttBwdArgs& a, cudaStream_t st) {
  using C = AttBwdCfg<D, MODE>;
  static bool attr = false;
  if (!attr) {
    if (cudaFuncSetAttribute(attention_bwd_kernel<D, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::BYTES) !=
        cudaSuccess)
      return -11;
    attr = true;
  }
  const long long blocks =
      static_cast<long long>(((C::ROWQ ? a.Sq : a.Skv) + AB_ROWS - 1) / AB_ROWS) * (C::ROWQ ? a.Hq : a.Hkv) * a.B;
  if (blocks > 0x7fffffffLL) return -2;
  attention_bwd_kernel<D, MODE><<<static_cast<unsigned>(blocks), AB_THREADS, C::BYTES, st>>>(a1, a2, b1, b2, o1, ov, a);
  return static_cast<int>(cudaGetLastError());
}

// q, o, d_o: bf16 [B, Sq, Hq, D]; k, v: bf16 [B, Skv, Hkv, D]; lse: fp32 [B, Hq, Sq] from the forward.
// Scratch: delta fp32 [B, Hq, Sq].
// Outputs: dq bf16 [B, Sq, Hq, D]; dk, dv bf16 [B, Skv, Hkv, D] (summed over the query heads of each GQA group).
extern "C" int cvb_attention_bwd(const void* q, const void* k, const void* v, const void* o, const void* d_o,
                                 const float* lse, float* delta, void* dq, void* dk, void* dv, long long B, int Sq,
                                 int Skv, int Hq, int Hkv, int D, float scale, int causal, long long q_pos0,
                                 long long k_pos0, int* status, void* stream) {
  if (B <= 0 || Sq <= 0 || Skv <= 0) return 0;
  if (Hkv <= 0 || Hq % Hkv || !(scale > 0.f) || (D != 128 && D != 256)) return -1;
  if (B * Sq > 0x7fffffffLL || B * Skv > 0x7fffffffLL) return -2;
  for (const void* p : {q, k, v, o, d_o, static_cast<const void*>(dq), static_cast<const void*>(dk),
                        static_cast<const void*>(dv)})
    if (reinterpret_cast<uintptr_t>(p) & 15) return -3;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const uint64_t qc = static_cast<uint64_t>(Hq) * D, kc = static_cast<uint64_t>(Hkv) * D;
  auto map = [&](CUtensorMap* m, const void* p, bool query, uint32_t box) {
    const uint64_t cols = query ? qc : kc, rows = query ? Sq : Skv;
    return make_tensor_map_3d(m, p, 2, cols, rows, B, cols * 2, cols * 2 * rows, 64, box);
  };
  CUtensorMap q128, q64, k128, k64, v128, v64, do128, do64, mdq, mdk, mdv;
  if (map(&q128, q, true, 128) || map(&q64, q, true, 64) || map(&do128, d_o, true, 128) || map(&do64, d_o, true, 64) ||
      map(&k128, k, false, 128) || map(&k64, k, false, 64) || map(&v128, v, false, 128) || map(&v64, v, false, 64) ||
      map(&mdq, dq, true, 128) || map(&mdk, dk, false, 128) || map(&mdv, dv, false, 128))
    return -10;
  const long long rows = B * Sq * Hq;
  attention_delta_kernel<<<static_cast<unsigned>((rows + 8 * DELTA_ROWS - 1) / (8 * DELTA_ROWS)), 256, 0, st>>>(
      static_cast<const __nv_bfloat16*>(o), static_cast<const __nv_bfloat16*>(d_o), delta, rows, Sq, Hq, D);
  AttBwdArgs a{};
  a.lse = lse; a.delta = delta; a.Sq = Sq; a.Skv = Skv; a.Hq = Hq; a.Hkv = Hkv; a.B = static_cast<int>(B);
  a.scale = scale; a.scale_log2 = scale * 1.4426950408889634f; a.causal = causal; a.q_pos0 = q_pos0; a.k_pos0 = k_pos0;
  a.status = status;
  int rc;
  if (D == 128) {
    rc = launch_bwd<128, BWD_KV>(k128, v128, q64, do64, mdk, mdv, a, st);
    if (rc == 0) rc = launch_bwd<128, BWD_Q>(q128, do128, k64, v64, mdq, mdq, a, st);
  } else {
    rc = launch_bwd<256, BWD_V>(k128, v128, q64, do64, mdv, mdv, a, st);
    if (rc == 0) rc = launch_bwd<256, BWD_K>(k128, v128, q64, do64, mdk, mdk, a, st);
    if (rc == 0) rc = launch_bwd<256, BWD_Q>(q128, do128, k64, v64, mdq, mdq, a, st);
  }
  return rc;
}
