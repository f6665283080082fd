// attn_decode.cuh — the attention block of a decode step for one (row, kv head, context slice),
// as a device function shared by the stand-alone kernel (attn_decode.cu: one CTA per item, the
// slices of a pair forming a thread-block cluster) and the resident decode kernel
// (decode_resident.cu: 128 threads of a resident CTA work through a list of items).
//
// The caller supplies an environment:
//   tid()            0..127, the thread's index among the 128 threads that run the item
//   sync_cta()       barrier among those 128 threads
//   kPush            keys and values come by TMA, and the slices' partial results are PUSHED (st.async, counted by an
//                    mbarrier) into a landing area (landing(), attn_dec_landing_bytes() of shared memory that nothing
//                    else uses) of the cluster CTA that finishes them: one way across the cluster, and nobody waits for
//                    a reader.  The slice's number is the CTA's rank in its cluster, and a CTA runs one item.
//   map_k, map_v     kPush: tensor maps of the caches as rows of d values, boxes of attn_dec_keys(d) rows of 64
//                    Without kPush 16-byte copies bring the keys and values, and the finishing CTA reads the partials
//                    where they lie, behind two barriers:
//   sync_group()     barrier among the CTAs that hold the slices of one (row, kv head),
//                    including a barrier among each CTA's own 128 threads
//   cluster_rank(s)  cluster rank of the CTA that holds slice s
//   kRows            the item is a row of AttnDecArgs::rows: its own slot and position, neighbouring pairs
//                    rotated, norms over all heads at once, a sink
//   settle(pos)      called once the first K/V tiles have been requested with a position that may
//                    be one step old: waits for whatever the caller's inputs depend on and returns
//                    the position to use (cached keys never change, so an early request is either
//                    right or is repeated)
//
// What bounds an item is its chain of dependent steps and the instructions of its few warps, not its bytes (a few MB per
// layer over all items).  So gains, angles and the first tiles are asked for before the projection is waited for; one
// round of loads then brings every vector of the new token, a warp per vector, with its norm in shuffles and its
// rotation pairs in one lane; the new token takes its place among the keys of a chunk instead of being a chunk of
// its own; a tile is asked for by one lane; P V is taken as O^T = V^T P^T, whose 8 heads fill the MMA's 8
// columns (half the instructions and registers of the other form, whose 16 rows they half fill); and nothing divides
// where a reciprocal does.  From a per-warp timeline: a soft-capped chunk spent 2100 of its 5100 cycles in divisions, a
// head norm 3000, the merge of 16 unrolled slices up to 2700.  Us that a launch keeps the stream, before / now: 32 rows
// of 530 keys, 8 kv heads of 128: 40.5 / 26; 4 x 2080, 4 of 256, soft-cap: 21 / 13; 8 x 1050, 4 of 128, 8 heads each:
// 16.7 / 9; 1 x 350, the same: 13.5 / 8.4; 8 x 576, 8 of 64: 7.0 / 5.4.
#pragma once

#include "kernels.h"
#include "mma.cuh"
#include "tc_common.cuh"

namespace cg {

constexpr int ATTN_MAX_REP = 8;  // query heads per kv head: rows 0..7 of the 16-row MMA tile

__device__ __forceinline__ float attn_ld_dsmem(uint32_t local_addr, uint32_t rank) {
  uint32_t remote;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local_addr), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
  return v;
}
// W = 1, 2 or 4 neighbouring floats through L2 (in the resident kernel another CTA wrote them in the same launch)
template <int W>
__device__ __forceinline__ void attn_ldcg(const float* p, float* v) {
  if constexpr (W == 1) {
    v[0] = __ldcg(p);
  } else if constexpr (W == 2) {
    const float2 x = __ldcg((const float2*)p);
    v[0] = x.x; v[1] = x.y;
  } else {
    const float4 x = __ldcg((const float4*)p);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
  }
}

// Keys per warp tile: 32, or 16 for head size 256 so that a CTA's tiles fit a third of an SM's shared memory.
__host__ __device__ constexpr int attn_dec_keys(int D) { return D > 128 ? 16 : 32; }

// shared memory one item needs (from a multiple of 1024 bytes): 8 query rows, a key and a value tile per warp, the new
// key and value, reductions and the tiles' barriers
template <int D>
__host__ __device__ constexpr size_t attn_dec_smem_bytes() {
  return (size_t)(8 * attn_dec_keys(D) * D + 8 * (D + 8) + 2 * D) * 2 + (size_t)(8 * ATTN_MAX_REP + 4) * 4 + 64;
}

// landing area of the push form: a barrier, {max, sum} per source slice and head, and per source slice its share of
// the output values that the CTA finishes
__host__ __device__ constexpr size_t attn_dec_landing_bytes(int rep, int d, int splits) {
  return 16 + (size_t)splits * ATTN_MAX_REP * 8 + (size_t)rep * d * 4;
}

template <int D, class Env>
__device__ __forceinline__ void attn_dec_item(const AttnDecArgs& a, float scale, int kvh, int64_t b, int split, int64_t pos_early,
                                              uint8_t* smem, Env& env) {
  constexpr int KT = attn_dec_keys(D);
  constexpr int MAX_REP = ATTN_MAX_REP;
  constexpr int LD = D + 8;     // padded rows of the queries: conflict-free ldmatrix
  constexpr int BOX = KT * 128; // bytes of a box of a tile: KT rows of 64 values
  constexpr int CH = D / 8;     // 16-byte chunks per row
  constexpr int W = D / 64;     // rotation pairs per lane
  constexpr int NV = 3;         // vectors of the new token per warp: at most 8 query heads, a key and a value on 4 warps
  constexpr int LDO = D + 4;    // row stride of the warps' outputs: conflict-free stores of O^T fragments
  // Tiles are D / 64 boxes of KT rows of 64 values; 16-byte chunk c of row r of a box lies at place c ^ (r & 7), as TMA's
  // 128-byte swizzle has it (the tiles begin on a multiple of 1024 bytes): conflict-free ldmatrix
  uint8_t* kt = smem;                                    // [4 warps] key tiles
  uint8_t* vt = kt + 4 * KT * D * 2;                     // [4 warps] value tiles
  __nv_bfloat16* qt = (__nv_bfloat16*)(vt + 4 * KT * D * 2);  // [8][LD] query heads (rows >= rep are zero)
  __nv_bfloat16* knew = qt + 8 * LD;                     // [D] the new key
  __nv_bfloat16* vnew = knew + D;                        // [D]
  float* red_m = (float*)(vnew + D);                     // [4][MAX_REP]
  float* red_l = red_m + 4 * MAX_REP;                    // [4][MAX_REP]
  volatile int* cta_abort = (volatile int*)(red_l + 4 * MAX_REP);
  float* red_o = (float*)kt;                             // [4][MAX_REP][LDO] f32, over the tiles after the loop

  const int tid = env.tid(), warp = tid >> 5, lane = tid & 31;
  // this warp's barriers: its keys have arrived, its values have arrived
  const uint32_t bar_k = (uint32_t)__cvta_generic_to_shared(red_l + 4 * MAX_REP + 4) + (uint32_t)warp * 16u, bar_v = bar_k + 8;
  if constexpr (Env::kPush) {
    if (lane == 0) {
      tc::mbar_init(bar_k, 1);
      tc::mbar_init(bar_v, 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    if (tid == 0) *cta_abort = 0;  // (for the other warps behind the first CTA barrier)
  }
  const int rep = a.nh / a.nkv;
  const int S = a.splits;
  // A CTA finishes `wide` neighbouring columns of every head.  Landing area of the push form: slice s's {max, sum} of
  // head r at land_ml[s][r], its values of those outputs at land_o[s][r].
  const int lg = __ffs(S) - 1, wide = D >> lg;  // (the slices are a power of two in number)
  const int per = rep * wide, lgw = 31 - __clz(wide);
  uint32_t land_bar = 0, land_ml = 0, land_o = 0;
  if constexpr (Env::kPush) {
    land_bar = (uint32_t)__cvta_generic_to_shared(env.landing());
    land_ml = land_bar + 16;
    land_o = land_ml + (uint32_t)(S * MAX_REP * 8);
    if (S > 1) {
      if (tid == 0) {
        tc::mbar_init(land_bar, 1);
        tc::mbar_expect_tx(land_bar, (uint32_t)(rep * D * 4 + S * rep * 8));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      }
      // the peers' barriers exist once they have arrived here; waited for just before the pushes
      __syncwarp();
      asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    }
  }
  // pos: position of the new token = number of cached keys
  int64_t place = b;
  bool in_range = true;
  if constexpr (Env::kRows) {
    place = a.rows.slot[b];
    if (place < 0 || (place + 1) * a.nkv * a.Tmax > a.cache_rows) {
      *a.err = DEV_INDEX;
      place = 0;
      in_range = false;
    }
  }
  __nv_bfloat16* kbase = a.k_cache + ((place * a.nkv + kvh) * a.Tmax) * (int64_t)D;
  __nv_bfloat16* vbase = a.v_cache + ((place * a.nkv + kvh) * a.Tmax) * (int64_t)D;

  // The visible keys are the kf kept first ones, [lo, pos) and the new one.  They are numbered in that order, with the
  // numbers from kf to the next multiple of KT left out; the new one is number `fresh`; [t0, t1) is this CTA's slice.
  int64_t pos = pos_early;
  int t0 = 0, t1 = 0, kf = 0, kfp = 0, fresh = 0;
  int64_t skip = 0;  // from a key's number to its place in the cache, behind the kept ones
  auto plan = [&]() {
    const int64_t lo = a.window > 0 ? max((int64_t)0, pos - a.window + 1) : 0;
    if constexpr (Env::kRows) {
      kf = (int)min(a.keep_first, lo);
      kfp = (kf + KT - 1) / KT * KT;
    }
    skip = lo - kfp;
    fresh = (int)(pos - skip);
    int n = (fresh + S) >> lg;
    n = (n + KT - 1) / KT * KT;
    t0 = split * n;
    t1 = min(fresh + 1, t0 + n);
  };
  plan();

  uint8_t* kw = kt + warp * (KT * D * 2);
  uint8_t* vw = vt + warp * (KT * D * 2);
  const uint32_t kw_u = (uint32_t)__cvta_generic_to_shared(kw);
  const uint32_t vw_u = (uint32_t)__cvta_generic_to_shared(vw);
  const uint32_t qt_u = (uint32_t)__cvta_generic_to_shared(qt);

  // Request the first chunk of this warp now: it does not depend on q.  One lane asks for a tile by D / 64 TMA loads of
  // whole boxes (16-byte copies cost a third of the kernel's instructions, which a warp has little to hide behind; bulk
  // copies of single rows are slower than those where rows are 128 bytes).  Keys and values have barriers of their
  // own: the next keys are asked for as soon as the scores have been taken, the next values behind the
  // product, so that of a warp's two tiles one is always on its way.
  auto request = [&](int c0, bool keys) {
    if constexpr (Env::kPush) {
      if (c0 < t1 && lane == 0) {
        const uint32_t bar = keys ? bar_k : bar_v, tile = keys ? kw_u : vw_u;
        const int at = (int)((place * a.nkv + kvh) * a.Tmax + (c0 < kfp ? c0 : c0 + skip));
        tc::mbar_expect_tx(bar, KT * D * 2);
#pragma unroll
        for (int x = 0; x < D / 64; ++x) tc::tma_load_2d(tile + x * BOX, keys ? env.map_k : env.map_v, x * 64, at, bar);
      }
    } else {
      if (c0 < t1) {
        const uint32_t tile = keys ? kw_u : vw_u;
        const __nv_bfloat16* from = keys ? kbase : vbase;
#pragma unroll 4
        for (int i = lane; i < KT * CH; i += 32) {
          const int r = i / CH, ch = i % CH;
          const int64_t key = c0 + r + skip;
          const bool ok = key < pos;
          cp_async16(tile + (uint32_t)((ch >> 3) * BOX + r * 128 + (((ch & 7) ^ (r & 7)) << 4)), from + (ok ? key : 0) * D + ch * 8, ok ? 16 : 0);
        }
      }
      cp_async_commit();
    }
  };
  uint32_t phase = 0;  // of both barriers
  int c0 = t0 + warp * KT;
  request(c0, true);
  request(c0, false);

  // Warp w has the new token's vectors w, w + 4, w + 8: the query heads, the key, the value.  A lane holds both
  // components of W rotation pairs.  Pairs are (j, j + D / 2) with j = lane * W + i, or neighbours with j = lane + 32 i.
  const int heads = a.nh + 2 * a.nkv;
  auto pair = [&](int i) { return Env::kRows ? lane + 32 * i : lane * W + i; };
  auto head_of = [&](int id) { return id < rep ? kvh * rep + id : id == rep ? a.nh + kvh : a.nh + a.nkv + kvh; };
  auto is_new = [&](int v) { return warp + 4 * v < rep + 2; };
  // what does not depend on the projection: gains and angles
  float g1[NV][W], g2[NV][W], cs[W], sn[W], temp = 1.f;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int id = warp + 4 * v;
#pragma unroll
    for (int i = 0; i < W; ++i) g1[v][i] = g2[v][i] = 1.f;
    if (a.q_gamma && id <= rep) {
      if constexpr (Env::kRows) {
        const float* g = id < rep ? a.q_gamma + (int64_t)(kvh * rep + id) * D : a.k_gamma + (int64_t)kvh * D;
#pragma unroll
        for (int i = 0; i < W; ++i) {
          const float2 x = *((const float2*)g + pair(i));
          g1[v][i] = x.x; g2[v][i] = x.y;
        }
      } else {
        const float* g = id < rep ? a.q_gamma : a.k_gamma;
        const float plus = a.norm_plus_one ? 1.f : 0.f;
#pragma unroll
        for (int i = 0; i < W; ++i) {
          g1[v][i] = plus + g[pair(i)];
          g2[v][i] = plus + g[pair(i) + D / 2];
        }
      }
    }
  }
  auto angles = [&]() {
    const int n = Env::kRows ? a.rot_dims / 2 : D / 2;
#pragma unroll
    for (int i = 0; i < W; ++i) {
      const int j = pair(i);
      cs[i] = 1.f; sn[i] = 0.f;
      if (j < n) { cs[i] = a.cos_t[pos * n + j]; sn[i] = a.sin_t[pos * n + j]; }
    }
    if constexpr (Env::kRows)
      if (a.q_temp) temp = a.q_temp[pos];
  };
  angles();
  for (int i = tid; i < (8 - rep) * CH; i += 128) *(uint4*)(qt + (rep + i / CH) * LD + i % CH * 8) = make_uint4(0u, 0u, 0u, 0u);
  bool ok = true;
  {
    int64_t pos_now = env.settle(pos);
    if constexpr (Env::kPush)
      if ((uint64_t)pos_now >= (uint64_t)a.Tmax) {
        *a.err = DEV_INDEX;
        pos_now = pos;
        in_range = false;
      }
    if (pos_now != pos) {  // the early position was stale: let the copies land, then ask again
      if constexpr (Env::kPush) {
        if (c0 < t1) {
          int gave_up = 0;
          ok = tc::mbar_wait(bar_k, phase, &gave_up, a.err) && tc::mbar_wait(bar_v, phase, &gave_up, a.err);
          ok = __all_sync(0xffffffffu, ok) != 0;
          if (!ok) {
            tc::mbar_drain(bar_k, phase, a.err);
            tc::mbar_drain(bar_v, phase, a.err);
          }
          phase ^= 1u;
        }
      } else {
        cp_async_wait_group<0>();
      }
      __syncwarp();
      pos = pos_now;
      plan();
      c0 = t0 + warp * KT;
      if (ok) {
        request(c0, true);
        request(c0, false);
      }
      angles();
    }
  }

  // ---- 1. q, k, v of the new token ----
  int64_t ld_row = (int64_t)heads * D, ld_out = (int64_t)a.nh * D;
  if constexpr (Env::kRows) {
    if (a.ld_qkv) ld_row = a.ld_qkv;
    if (a.ld_out) ld_out = a.ld_out;
  }
  const float* row = a.qkv + b * ld_row;
  {
    float x1[NV][W], x2[NV][W];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
#pragma unroll
      for (int i = 0; i < W; ++i) x1[v][i] = x2[v][i] = 0.f;
      if (!is_new(v)) continue;
      const float* src = row + (int64_t)head_of(warp + 4 * v) * D;
      if constexpr (Env::kRows) {
#pragma unroll
        for (int i = 0; i < W; ++i) {
          const float2 x = __ldcg((const float2*)src + pair(i));
          x1[v][i] = x.x; x2[v][i] = x.y;
        }
      } else {
        attn_ldcg<W>(src + lane * W, x1[v]);
        attn_ldcg<W>(src + lane * W + D / 2, x2[v]);
      }
    }
    if (Env::kRows && a.q_gamma) {
      // norms over all query heads and over all key heads
      float ss[2] = {0.f, 0.f};
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        const float4* src = (const float4*)(row + (part ? (int64_t)a.nh * D : 0));
        const int n = (part ? a.nkv : a.nh) * D / 4;
#pragma unroll 4
        for (int i = tid; i < n; i += 128) {
          const float4 v = __ldcg(src + i);
          ss[part] += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
        }
      }
#pragma unroll
      for (int o = 16; o; o >>= 1) {
        ss[0] += __shfl_xor_sync(0xffffffffu, ss[0], o);
        ss[1] += __shfl_xor_sync(0xffffffffu, ss[1], o);
      }
      if (lane == 0) { red_m[warp] = ss[0]; red_m[4 + warp] = ss[1]; }
      env.sync_cta();
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const int id = warp + 4 * v;
        if (id > rep) continue;
        const float* r = red_m + (id < rep ? 0 : 4);
        const float f = 1.f / sqrtf(((r[0] + r[1]) + (r[2] + r[3])) / (float)((id < rep ? a.nh : a.nkv) * a.norm_dim) + a.norm_eps);
#pragma unroll
        for (int i = 0; i < W; ++i) { x1[v][i] *= f * g1[v][i]; x2[v][i] *= f * g2[v][i]; }
      }
    } else if (Env::kRows ? a.head_norm != 0 : a.q_gamma != nullptr) {
      // norms per head
      float ss[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        ss[v] = 0.f;
#pragma unroll
        for (int i = 0; i < W; ++i) ss[v] += x1[v][i] * x1[v][i] + x2[v][i] * x2[v][i];
      }
#pragma unroll
      for (int o = 16; o; o >>= 1)
#pragma unroll
        for (int v = 0; v < NV; ++v) ss[v] += __shfl_xor_sync(0xffffffffu, ss[v], o);
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        if (warp + 4 * v > rep) continue;
        if constexpr (Env::kRows) {
          const float f = 1.f / sqrtf(ss[v] / (float)a.norm_dim + a.norm_eps);
#pragma unroll
          for (int i = 0; i < W; ++i) { x1[v][i] *= f; x2[v][i] *= f; }
        } else {
          const float f = 1.f / sqrtf(ss[v] * (1.f / D) + a.norm_eps);
#pragma unroll
          for (int i = 0; i < W; ++i) { x1[v][i] *= f * g1[v][i]; x2[v][i] *= f * g2[v][i]; }
        }
      }
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      if (!is_new(v)) continue;
      const int id = warp + 4 * v;
      if (id <= rep) {
        const float t = id < rep ? temp : 1.f;
#pragma unroll
        for (int i = 0; i < W; ++i) {
          const float u = x1[v][i], w = x2[v][i];
          if (!Env::kRows || pair(i) < a.rot_dims / 2) {
            x1[v][i] = cs[i] * u - sn[i] * w;
            x2[v][i] = cs[i] * w + sn[i] * u;
          }
          x1[v][i] *= t; x2[v][i] *= t;
        }
      }
      auto put = [&](__nv_bfloat16* to) {
#pragma unroll
        for (int i = 0; i < W; ++i) {
          const int j = pair(i);
          if constexpr (Env::kRows) {
            *(__nv_bfloat162*)(to + 2 * j) = __floats2bfloat162_rn(x1[v][i], x2[v][i]);
          } else {
            to[j] = __float2bfloat16_rn(x1[v][i]);
            to[j + D / 2] = __float2bfloat16_rn(x2[v][i]);
          }
        }
      };
      put(id < rep ? qt + id * LD : id == rep ? knew : vnew);
      if (id >= rep && split == 0 && in_range) put((id == rep ? kbase : vbase) + pos * D);  // append to the cache for the following steps
    }
  }
  env.sync_cta();
  if (!ok) {  // without keys from here on, but past every barrier
    *cta_abort = 1;
    c0 = t1;
  }

  // ---- 2. this warp's chunks of KT keys: S = Q K^T, online softmax, O^T += V^T P^T ----
  // In S a thread owns head hr = lane / 4 and, per 8-key tile, the two keys cq + {0, 1}; in O^T the two heads
  // cq + {0, 1} and, per 16 output columns, columns lane / 4 and 8 + lane / 4.
  const int hr = lane >> 2, cq = (lane & 3) * 2;
  const float* bias = nullptr;
  if constexpr (Env::kRows)
    if (a.bias && hr < rep) bias = a.bias + (int64_t)(kvh * rep + hr) * a.ld_bias;
  float m = -INFINITY, l = 0.f;
  float o[D / 16][4];
#pragma unroll
  for (int j = 0; j < D / 16; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
  // c tanh(x / c) = c (2 / (1 + 2^(x cap_unit / scale)) - 1)
  const float cap_unit = a.softcap > 0.f ? -2.f * 1.44269504088896340736f * scale / a.softcap : 0.f;
  auto chunk_of = [&](uint8_t* tile, int r, int ch) {
    return (uint4*)(tile + (ch >> 3) * BOX + r * 128 + (((ch & 7) ^ (r & 7)) << 4));
  };
  // the new token's row of a tile, once the copies have landed
  auto insert = [&](uint8_t* tile, const __nv_bfloat16* from) {
    const int r = fresh - c0;
    if (r >= 0 && r < KT) {
      for (int i = lane; i < CH; i += 32) *chunk_of(tile, r, i) = *(const uint4*)(from + i * 8);
      __syncwarp();
    }
  };
  // ldmatrix addresses of this lane: rows (lane & 7) + 8 (lane / 16) of a tile, chunks 2 x + (lane / 8) % 2 of a box
  const uint32_t qa = qt_u + (uint32_t)((lane & 7) * LD + (lane >> 3) * 8) * 2u;
  uint32_t xa[4];
#pragma unroll
  for (int x = 0; x < 4; ++x)
    xa[x] = kw_u + (uint32_t)(((lane & 7) + 8 * (lane >> 4)) * 128 + (((2 * x + ((lane >> 3) & 1)) ^ (lane & 7)) << 4));
  const uint32_t to_v = vw_u - kw_u;
  // A warp leaves the loop as a whole where a wait gave up, behind the copies that are on their way to it.
  auto landed = [&](uint32_t bar) {
    if constexpr (Env::kPush) return __all_sync(0xffffffffu, tc::mbar_wait(bar, phase, cta_abort, a.err)) != 0;
    cp_async_wait_group<1>();
    __syncwarp();
    return true;
  };
  for (; c0 < t1; c0 += 4 * KT) {
    const int live = (c0 < kfp ? kf : t1) - c0;  // keys of this chunk, at least one
    if (!landed(bar_k)) {
      tc::mbar_drain(bar_k, phase, a.err);
      tc::mbar_drain(bar_v, phase, a.err);
      break;
    }
    insert(kw, knew);
    // (two sums per key tile: a chain of half the length)
    float s[KT / 8][4], s2[KT / 8][4];
#pragma unroll
    for (int j = 0; j < KT / 8; ++j) s[j][0] = s[j][1] = s[j][2] = s[j][3] = s2[j][0] = s2[j][1] = s2[j][2] = s2[j][3] = 0.f;
#pragma unroll
    for (int kk = 0; kk < D / 16; kk += 2) {
      uint32_t q[4];
      ldsm_x4(qa + (uint32_t)(kk * 32), q[0], q[1], q[2], q[3]);
#pragma unroll
      for (int j = 0; j < KT / 8; j += 2) {
        uint32_t b0, b1, b2, b3;
        ldsm_x4(xa[kk & 3] + (uint32_t)(j * 8 * 128 + kk / 4 * BOX), b0, b1, b2, b3);
        mma_bf16(s[j], q[0], 0u, q[1], 0u, b0, b1);
        mma_bf16(s[j + 1], q[0], 0u, q[1], 0u, b2, b3);
        ldsm_x4(xa[(kk + 1) & 3] + (uint32_t)(j * 8 * 128 + kk / 4 * BOX), b0, b1, b2, b3);
        mma_bf16(s2[j], q[2], 0u, q[3], 0u, b0, b1);
        mma_bf16(s2[j + 1], q[2], 0u, q[3], 0u, b2, b3);
      }
    }
    __syncwarp();
    request(c0 + 4 * KT, true);
    // scale, soft-cap, mask; this head's maximum over the chunk
    float mx = -INFINITY;
#pragma unroll
    for (int j = 0; j < KT / 8; ++j) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float v = s[j][e] + s2[j][e];
        v = a.softcap > 0.f ? a.softcap * fmaf(2.f, rcp_newton(1.f + fast_exp2(v * cap_unit)), -1.f) : v * scale;
        const int key = c0 + j * 8 + cq + e;
        const bool keep = key - c0 < live;
        if constexpr (Env::kRows)
          if (bias && keep && key < fresh)   // (at the new token itself the distance is 0, and so is what is taken off)
            v -= bias[pos - (key < kfp ? key : key + skip)];
        v = keep ? v : -INFINITY;
        s[j][e] = v;
        mx = fmaxf(mx, v);
      }
    }
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const float mnew = fmaxf(m, mx);  // finite: the first key of every chunk is live
    const float corr = __expf(m - mnew);
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < KT / 8; ++j) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float p = __expf(s[j][e] - mnew);
        s[j][e] = p;
        sum += p;
      }
    }
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    l = l * corr + sum;
    const float m_old = m;
    m = mnew;
    if (__any_sync(0xffffffffu, corr != 1.f && m_old != -INFINITY)) {  // (a factor of one changes nothing, nor does one on zeros)
      const float f0 = __shfl_sync(0xffffffffu, corr, cq * 4), f1 = __shfl_sync(0xffffffffu, corr, cq * 4 + 4);
#pragma unroll
      for (int j = 0; j < D / 16; ++j) {
        o[j][0] *= f0; o[j][1] *= f1;
        o[j][2] *= f0; o[j][3] *= f1;
      }
    }
    if (!landed(bar_v)) {
      tc::mbar_drain(bar_v, phase, a.err);
      if (c0 + 4 * KT < t1) tc::mbar_drain(bar_k, phase ^ 1u, a.err);
      break;
    }
    insert(vw, vnew);
    if (live < KT) {  // probability zero times whatever lies behind the live rows must not be NaN
      for (int i = lane; i < (KT - live) * CH; i += 32) *chunk_of(vw, live + i / CH, i % CH) = make_uint4(0u, 0u, 0u, 0u);
      // (behind kept first keys the tile is loaded again: TMA's writes come after these)
      if constexpr (Env::kPush && Env::kRows)
        if (c0 + 4 * KT < t1) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    // O^T += V^T P^T: the scores' fragments are those of P^T
#pragma unroll
    for (int kk = 0; kk < KT / 16; ++kk) {
      const uint32_t b0 = pack_bf16(s[2 * kk][0], s[2 * kk][1]);
      const uint32_t b1 = pack_bf16(s[2 * kk + 1][0], s[2 * kk + 1][1]);
#pragma unroll
      for (int j = 0; j < D / 16; ++j) {
        uint32_t a0, a1, a2, a3;
        ldsm_x4_t(xa[j & 3] + to_v + (uint32_t)(kk * 16 * 128 + j / 4 * BOX), a0, a1, a2, a3);
        mma_bf16(o[j], a0, a1, a2, a3, b0, b1);
      }
    }
    __syncwarp();
    request(c0 + 4 * KT, false);
    phase ^= 1u;
  }

  // ---- 3. merge the four warps in this CTA, then the slices across the cluster ----
  if ((lane & 3) == 0) red_m[warp * MAX_REP + hr] = m;
  env.sync_cta();  // all tiles are dead: reuse their space
  // the maximum over the warps, to which each brings its sums and outputs
  auto top_of = [&](int r) { return fmaxf(fmaxf(red_m[r], red_m[MAX_REP + r]), fmaxf(red_m[2 * MAX_REP + r], red_m[3 * MAX_REP + r])); };
  auto factor = [&](int r) {
    const float mw = red_m[warp * MAX_REP + r];
    return mw == -INFINITY ? 0.f : __expf(mw - top_of(r));
  };
  auto sum_of = [&](int r) { return (red_l[r] + red_l[MAX_REP + r]) + (red_l[2 * MAX_REP + r] + red_l[3 * MAX_REP + r]); };
  if ((lane & 3) == 0) red_l[warp * MAX_REP + hr] = l * factor(hr);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int r = cq + h;
    if (r < rep) {
      const float f = factor(r);
      float* to = red_o + (warp * MAX_REP + r) * LDO + hr;
#pragma unroll
      for (int j = 0; j < D / 16; ++j) {
        to[j * 16] = o[j][h] * f;
        to[j * 16 + 8] = o[j][2 + h] * f;
      }
    }
  }
  // the merged output oo over the merged sum ll of exp(score - mm), which the sink joins, gated and scaled
  auto finished = [&](int r, int e, float mm, float ll, float oo) {
    if constexpr (Env::kRows) {
      oo *= a.out_scale;
      if (a.gate) oo *= 1.f / (1.f + __expf(-__ldcg(a.gate + b * a.ld_gate + (a.wide_gate ? (kvh * rep + r) * D + e : kvh * rep + r))));
      if (a.sink) {
        const float sk = a.sink[kvh * rep + r], top = fmaxf(mm, sk);
        const float f = __expf(mm - top);
        return oo * f / (ll * f + __expf(sk - top));
      }
    }
    return ll > 0.f ? oo / ll : 0.f;
  };
  auto store = [&](int r, int e, float v) { a.out[b * ld_out + (kvh * rep + r) * (int64_t)D + e] = __float2bfloat16_rn(v); };
  // four neighbouring outputs, added over the warps in order
  auto four = [&](int r, int e) {
    float4 v = *(const float4*)(red_o + r * LDO + e);
#pragma unroll
    for (int w = 1; w < 4; ++w) {
      const float4 x = *(const float4*)(red_o + (w * MAX_REP + r) * LDO + e);
      v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
    }
    return v;
  };
  env.sync_cta();
  if (S == 1) {
    for (int i = tid * 4; i < rep * D; i += 512) {
      const int r = i / D, e = i % D;
      const float4 v = four(r, e);
      const float mm = top_of(r), ll = sum_of(r);
      store(r, e, finished(r, e, mm, ll, v.x));
      store(r, e + 1, finished(r, e + 1, mm, ll, v.y));
      store(r, e + 2, finished(r, e + 2, mm, ll, v.z));
      store(r, e + 3, finished(r, e + 3, mm, ll, v.w));
    }
    env.sync_cta();  // the partials are read: the next item of a resident CTA may reuse the space
    return;
  }
  // The slices of one (row, kv head) lie in one thread-block cluster.  (Kept as loops: every instruction of a step's
  // kernel is fetched anew, and 16 slices unrolled took 1000 to 2500 cycles here.)
  auto merge = [&](int r, int e, auto ml, auto ol) {
    float mm = -INFINITY;
#pragma unroll 4
    for (int s = 0; s < S; ++s) mm = fmaxf(mm, ml(s).x);
    float ll = 0.f, oo = 0.f;
#pragma unroll 4
    for (int s = 0; s < S; ++s) {
      const float2 x = ml(s);
      const float f = x.x == -INFINITY ? 0.f : __expf(x.x - mm);
      ll += x.y * f;
      oo += ol(s) * f;
    }
    store(r, e, finished(r, e, mm, ll, oo));
  };
  if constexpr (Env::kPush) {
    auto remote = [&](uint32_t addr, int rank) {
      uint32_t to;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(addr), "r"(rank));
      return to;
    };
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (tid < MAX_REP * S && (tid & (MAX_REP - 1)) < rep) {
      const int s = tid / MAX_REP, r = tid & (MAX_REP - 1);
      const float mm = top_of(r), ll = sum_of(r);
      asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::"r"(
                       remote(land_ml + (uint32_t)((split * MAX_REP + r) * 8), s)),
                   "r"(__float_as_uint(mm)), "r"(__float_as_uint(ll)), "r"(remote(land_bar, s))
                   : "memory");
    }
    for (int i = tid * 4; i < rep * D; i += 512) {
      const int r = i / D, e = i % D, owner = e >> lgw;
      const float4 v = four(r, e);
      asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                       remote(land_o + (uint32_t)((split * per + r * wide + (e & (wide - 1))) * 4), owner)),
                   "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)), "r"(__float_as_uint(v.z)), "r"(__float_as_uint(v.w)),
                   "r"(remote(land_bar, owner))
                   : "memory");
    }
    // Arrived when every CTA of the cluster has issued its pushes; waited for before this CTA leaves, so that no
    // push can find its target gone even where a wait has given up.
    __syncwarp();
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    if (tc::mbar_wait_cluster(land_bar, 0, cta_abort, a.err)) {
      const float* ml = env.landing() + 4;
      const float* ol = ml + S * MAX_REP * 2;
      for (int t = tid; t < per; t += 128) {
        const int r = t >> lgw;
        merge(r, split * wide + (t & (wide - 1)), [&](int s) { return *(const float2*)(ml + (s * MAX_REP + r) * 2); },
              [&](int s) { return ol[s * per + t]; });
      }
    }
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (*cta_abort) tc::mbar_drain(land_bar, 0, a.err);  // (issued is not arrived: what is still on its way, after a wait gave up)
  } else {
    // this slice's partial: {max, sum} and the values of every head, left in shared memory for the group
    float* part_ml = red_o + 4 * MAX_REP * LDO;  // [MAX_REP][2]
    float* part_o = part_ml + 2 * MAX_REP;       // [MAX_REP][D]
    for (int i = tid * 4; i < rep * D; i += 512) {
      const int r = i / D, e = i % D;
      if (e == 0) {
        part_ml[2 * r] = top_of(r);
        part_ml[2 * r + 1] = sum_of(r);
      }
      *(float4*)(part_o + i) = four(r, e);
    }
    env.sync_group();
    const uint32_t ml_u = (uint32_t)__cvta_generic_to_shared(part_ml);
    const uint32_t po_u = (uint32_t)__cvta_generic_to_shared(part_o);
    for (int t = tid; t < per; t += 128) {
      const int r = t >> lgw, e = split * wide + (t & (wide - 1));
      merge(r, e,
            [&](int s) {
              return make_float2(attn_ld_dsmem(ml_u + (uint32_t)(2 * r) * 4u, env.cluster_rank(s)),
                                 attn_ld_dsmem(ml_u + (uint32_t)(2 * r + 1) * 4u, env.cluster_rank(s)));
            },
            [&](int s) { return attn_ld_dsmem(po_u + (uint32_t)(r * D + e) * 4u, env.cluster_rank(s)); });
    }
    // nobody leaves while a peer may still read its shared memory
    env.sync_group();
  }
}

}  // namespace cg
