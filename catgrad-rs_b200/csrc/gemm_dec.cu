// gemm_dec.cu — the decode-step GEMM: y[M, N] = x[M, K] w[N, K]^T for M <= 32 tokens.
//
// With a handful of tokens the linear layers of catgrad-llm/src/models/llama.rs:12-115 are
// pure weight streaming, so this kernel is built around keeping HBM busy:
//
//   * warp 0 streams 128-row weight tiles by TMA into a shared-memory ring and starts doing
//     so BEFORE the preceding kernel has finished (programmatic dependent launch): weights
//     do not depend on it.  Only the small bf16 activation tiles wait for the predecessor.
//     Most CTAs find room only as their predecessors leave (median start of a CTA = end of the
//     preceding kernel, per-CTA timeline of a Llama-3.2-1B step), so the first requests go out as soon
//     as their barriers exist, ahead of the TMEM allocation and the CTA's first barrier.
//   * a CTA keeps its shared-memory ring small (about a third of an SM) so that the CTAs of
//     the NEXT GEMM in the stream can already be resident and prefetching their weights while
//     this one computes: the HBM stream does not stop at kernel boundaries.
//   * warp 1 issues tcgen05.mma (128 x TN x 16, f32 accumulators in TMEM).  For the gate/up
//     pair of the FFN both 128-row tiles share the CTA and the epilogue writes
//     act(gate) * up directly (llama.rs:27), so the [M, 2F] intermediate never exists.
//   * split-K partials are PUSHED over distributed shared memory inside a thread-block cluster:
//     every CTA stores its partial rows (st.async) into the exchange area of the CTA that finishes
//     them, whose own mbarrier counts the bytes, and the owner adds the partials in rank
//     order (deterministic) out of its own shared memory and applies the epilogue (residual add /
//     bf16 / act) once.  No CTA reads another's memory; the residual of the element a thread will
//     finish is fetched while the MMAs still run.
//   * every kernel of a step waits for the one before it, so what a single thread issues between two
//     arrivals is felt: slots and descriptors are counted along instead of divided and rebuilt (a
//     division by the runtime ring depth and four descriptors per stage had cost 4 % of a step), the
//     activations that follow the dependency are fetched by the idle epilogue warps, and TMEM is given
//     back beside the epilogue.
//     A step of the Llama-3.2-1B shape, batch 1 / batch 8: 733 / 835 us -> 645 / 754 us; four layers of
//     the Gemma-2-2B shape 514 -> 491 us, the Ralapel design 792 -> 740 us.  Of that the early requests and
//     the cheaper epilogue indices give 7 %.
//     The epilogue is bound by instructions of a few warps, not by bytes.  It has one form per kind of output,
//     a thread finishes one row and steps through the tokens by constants, only the splits there are get added,
//     sigmoids have no division, and the sums of squares of a handed-over norm are asked for together with the
//     activations instead of behind them.  From a per-CTA timeline (Llama-3.2-1B shape, batch 8): the norm's factors
//     3200 -> 900 cycles behind the activations, ahead of the accumulators now; a value's way from the last addend to
//     memory 1900 to 5800 -> 800 to 2200.  Ms per pass: Llama-3.2-1B shape, batch 8 101.2 -> 98.9, four layers
//     of the Llama-3-8B shape, batch 32 66.0 -> 61.8, Ralapel, batch 8 52.5 -> 50.6.
//
//   * two optional hand-overs ride on the epilogue.  Norm hand-over: a residual GEMM also
//     leaves bf16(out * gain) and per-CTA sums of out^2, and the GEMM behind the norm applies
//     1 / rms per row to its accumulators (RMSNorm(x) W^T = (x gain) W^T / rms(x)), so decode
//     steps of pre-norm models run no norm kernels.  Push: under tensor parallelism the partial
//     product goes straight into every rank's mapped exchange area and the last CTA raises
//     this rank's flag there (peer.cuh), instead of a collective call.
//
// All waits are bounded; on expiry the context's error word is raised and the kernel still
// passes its cluster barriers, frees its TMEM and returns.
#include <algorithm>
#include <type_traits>

#include "act.cuh"
#include "kernels.h"
#include "peer.cuh"
#include "tc_common.cuh"

namespace cg {

namespace {

using namespace tc;

struct DecArgs {
  void* out;
  int64_t ldo;
  const float* residual;
  int out_mode;
  int dual, act, up_off;
  int M, N, K;
  int kb_total, kb_per_split, splits, stages;
  int lg_rows_per;  // log2 of the rows of a tile that a split finishes (128 / splits)
  int x_rows;       // activation rows per k block in the ring (8 or TN)
  int xstage_cols;  // split-K: token columns of the exchange area (>= min(TN, M)); 0 without split-K
  int xstage_in_ring;  // the exchange area lies over the ring (more than 16 tokens: it would cost the ring a
                       // stage): then a first cluster barrier says every CTA's ring is idle before anyone pushes
  int32_t* err;
  int trace;  // slot in the timeline buffer, or -1
  const __nv_bfloat16* x;  // [M, K], leading dimension ldx
  int64_t ldx;
  PeerPush push;  // out_mode 3
  int total_ctas;
  // norm hand-over (see DecGemm): producer side ...
  __nv_bfloat16* xb_out;
  const float* g_next;
  int g_plus_one;
  float* ss_out;
  // ... and consumer side
  const float* ss_in;
  int ss_parts;
  float ss_inv_h, ss_eps;
};

constexpr int SS_FIRST = 4;      // partial sums of squares a thread asks for together with its activations
constexpr int SQ_FLOATS = 2048;  // per-CTA staging of squared outputs (cluster epilogue)

// Timeline of the decode GEMM launches (diagnostics): per slot {first CTA start, predecessor
// complete, last accumulator ready, last CTA end} in globaltimer nanoseconds.
constexpr int TRACE_SLOTS = 2048;
__device__ unsigned long long g_trace[TRACE_SLOTS * 4];

__device__ __forceinline__ void trace_min(int slot, int f) {
  if (slot >= 0) atomicMin(&g_trace[slot * 4 + f], (unsigned long long)globaltimer());
}
__device__ __forceinline__ void trace_max(int slot, int f) {
  if (slot >= 0) atomicMax(&g_trace[slot * 4 + f], (unsigned long long)globaltimer());
}

// What the epilogue does with a finished sum.  One form per kind of output, chosen once per CTA.
enum Form : int { FORM_F32, FORM_BF16, FORM_RESIDUAL, FORM_NORM, FORM_DUAL, FORM_PUSH };
template <class F>
__device__ __forceinline__ void with_form(const DecArgs& p, F f) {
  if (p.dual) f(std::integral_constant<int, FORM_DUAL>{});
  else if (p.xb_out) f(std::integral_constant<int, FORM_NORM>{});
  else if (p.out_mode == 2) f(std::integral_constant<int, FORM_RESIDUAL>{});
  else if (p.out_mode == 0) f(std::integral_constant<int, FORM_F32>{});
  else if (p.out_mode == 3) f(std::integral_constant<int, FORM_PUSH>{});
  else f(std::integral_constant<int, FORM_BF16>{});
}
// silu or tanh-gelu of g
__device__ __forceinline__ float act_of(int act, float g) {
  return over_one_plus(g, __expf(-(act == 0 ? g : 1.5957691216f * (g + 0.044715f * g * g * g))));
}
// Output (m, n), o = m * ldo + n; `res`: the residual there; `gain`: the next norm's at n.  Returns what the row's sum of
// squares gets.
template <int FORM>
__device__ __forceinline__ float finish(const DecArgs& p, int m, int n, int64_t o, float g, float u, uint32_t parity, const float* sc,
                                        float res, float gain) {
  if (p.ss_in) {  // the activations were handed over un-normalised: the row's 1 / rms goes here
    g *= sc[m];
    u *= sc[m];
  }
  if constexpr (FORM == FORM_NORM) {
    // residual epilogue that also prepares the next norm: the new residual in f32, its
    // gain-scaled bf16 copy for the next GEMM, and its square for the row's sum of squares
    const float r = g + res;
    ((float*)p.out)[o] = r;
    p.xb_out[o] = __float2bfloat16_rn(r * gain);
    return r * r;
  } else if constexpr (FORM == FORM_PUSH) {
    // this rank's addend goes into slot [parity][rank] of every rank's exchange area
    const int64_t slot = ((int64_t)parity * p.push.world + p.push.rank) * p.push.max_elems + o;
    for (int r = 0; r < p.push.world; ++r) p.push.data[r][slot] = g;
  } else if constexpr (FORM == FORM_DUAL) {
    g = act_of(p.act, g) * u;
    if (p.out_mode == 0) ((float*)p.out)[o] = g;
    else ((__nv_bfloat16*)p.out)[o] = __float2bfloat16_rn(g);
  } else if constexpr (FORM == FORM_F32) {
    ((float*)p.out)[o] = g;
  } else if constexpr (FORM == FORM_BF16) {
    ((__nv_bfloat16*)p.out)[o] = __float2bfloat16_rn(bf16_out(p.out_mode, g, p.residual, n));
  } else {
    ((float*)p.out)[o] = g + res;
  }
  return 0.f;
}
// the splits' partial sums in rank order, all loads first
template <int S>
__device__ __forceinline__ float add_ranks(const float* x, int step) {
  float v[S];
#pragma unroll
  for (int s = 0; s < S; ++s, x += step) v[s] = *x;
  float sum = 0.f;
#pragma unroll
  for (int s = 0; s < S; ++s) sum += v[s];
  return sum;
}

__device__ __forceinline__ void st_async(uint32_t addr, uint32_t v, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr), "r"(v), "r"(bar)
               : "memory");
}

// Activation chunks (16 bytes) of the first k blocks: chunk id = ((k block * x_rows) + row) * 8 + place.
// Rows past M are not read (they feed unused columns); places past K are zero.
constexpr int XCH = 4;
__device__ __forceinline__ void load_x_chunks(const DecArgs& p, int kb0, int id0, int chunks, int lg_rows, uint4* v) {
#pragma unroll
  for (int j = 0; j < XCH; ++j) {
    const int id = id0 + j * 128;
    const int t = id >> 3, r = t & ((1 << lg_rows) - 1);
    const int k = (kb0 + (t >> lg_rows)) * BK + (id & 7) * 8;
    v[j] = make_uint4(0u, 0u, 0u, 0u);
    if (id < chunks && r < p.M && k < p.K)
      asm volatile("ld.global.cg.v4.u32 {%0, %1, %2, %3}, [%4];"
                   : "=r"(v[j].x), "=r"(v[j].y), "=r"(v[j].z), "=r"(v[j].w)
                   : "l"(p.x + (int64_t)r * p.ldx + k)
                   : "memory");
  }
}
__device__ __forceinline__ void store_x_chunks(uint32_t xbase, uint32_t stage_bytes, int id0, int chunks, int lg_rows, const uint4* v) {
#pragma unroll
  for (int j = 0; j < XCH; ++j) {
    const int id = id0 + j * 128;
    if (id >= chunks) break;
    const int t = id >> 3, r = t & ((1 << lg_rows) - 1);
    const uint32_t a = xbase + (uint32_t)(t >> lg_rows) * stage_bytes + (uint32_t)r * 128u + (uint32_t)(((id & 7) ^ (r & 7)) << 4);
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v[j].x), "r"(v[j].y), "r"(v[j].z), "r"(v[j].w) : "memory");
  }
}

// OCC: CTAs per SM the register allocation must allow (the fewer registers a CTA holds, the
// sooner the CTAs of the NEXT kernels in the stream fit beside it and start fetching their weights)
template <int TN, int OCC>
__global__ void __launch_bounds__(192, OCC)
k_gemm_dec(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, DecArgs p) {
  // activation rows fetched per k block: TN, or 8 for up to 8 tokens (the MMA still reads TN rows;
  // the rows past the 8th are whatever follows in shared memory and feed only unused columns)
  const uint32_t X_TILE = (uint32_t)p.x_rows * BK * 2;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - raw);
  const int STAGES = p.stages;
  const uint32_t wbytes = p.dual ? 2 * A_BYTES : A_BYTES;
  const uint32_t stage_bytes = wbytes + X_TILE;
  // split-K exchange area [splits][(1 + dual) * xstage_cols][128 / splits] f32.  Up to 16 tokens it lies
  // behind the ring (not inside it: the other CTAs of the cluster write here while this CTA may
  // still be streaming); above, inside the ring, guarded by one more cluster barrier.
  const uint32_t xbytes = (uint32_t)((p.dual ? 2 : 1) * p.xstage_cols) * BM * 4u;
  const uint32_t xoff = p.xstage_in_ring ? 0u : STAGES * stage_bytes;
  const uint32_t boff = STAGES * stage_bytes + (p.xstage_in_ring ? 0u : xbytes);
  const uint32_t bars = base + boff;  // full[STAGES], empty[STAGES], accum
  const uint32_t bar_accum = bars + 16 * STAGES;
  const uint32_t bar_x = bar_accum + 16;  // split-K: every addend of this CTA's rows has arrived
  volatile uint32_t* tmem_slot = (volatile uint32_t*)(gen + boff + 16 * STAGES + 8);
  volatile int* cta_abort = (volatile int*)(gen + boff + 16 * STAGES + 12);
  float* sc = (float*)(gen + boff + 16 * 8 + 64);  // [32] per-token 1 / rms (consumer side), [4][32] the warps' sums
  // [SQ_FLOATS] squared outputs (producer side): in the ring, which is idle by then (only this
  // CTA touches its ring)
  float* sq = (float*)(gen + (p.xstage_in_ring ? xbytes : 0u));

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n0 = blockIdx.x * BM, split = blockIdx.z;
  const int kb0 = split * p.kb_per_split;
  const int nkb = min(p.kb_total, kb0 + p.kb_per_split) - kb0;
  const uint32_t ncols = p.dual ? 2 * TN : (TN < 32 ? 32 : TN);
  const bool cluster = p.splits > 1;
  if (tid == 0) trace_min(p.trace, 0);

  if (tid == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(bars + 8 * s, 2);             // full[s]: weight arrival + activation arrival
      mbar_init(bars + 8 * (STAGES + s), 1);  // empty[s]: one tcgen05.commit
    }
    mbar_init(bar_accum, 1);
    if (cluster) {
      // all 128 rows / splits rows of every split, M tokens of one or two accumulators
      mbar_init(bar_x, 1);
      mbar_expect_tx(bar_x, (uint32_t)((p.dual ? 2 : 1) * p.M) * BM * 4u);
    }
    *cta_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    // weights first, before this CTA is even set up: they depend neither on the preceding kernel nor on
    // TMEM, and a CTA that starts when its predecessors leave is waited for from here on
    for (int i = 0; i < min(nkb, STAGES); ++i) {
      const uint32_t full = bars + 8 * i;
      const uint32_t a = base + i * stage_bytes;
      const int k = (kb0 + i) * BK;
      mbar_expect_tx(full, wbytes);
      tma_load_2d(a, &map_w, k, n0, full);
      if (p.dual) tma_load_2d(a + A_BYTES, &map_w, k, p.up_off + n0, full);
    }
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_acc = *tmem_slot;
  // the peers' barriers exist once they have arrived here; waited for just before the pushes
  if (cluster && !p.xstage_in_ring) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");

  bool acc_ok = false;
  float res0 = 0.f, res1 = 0.f, gain = 0.f;  // split-K: residuals of the first two elements this thread will finish, their gain
  if (warp == 0) {
    if (lane == 0) {
      const int pre = min(nkb, STAGES);
      if (nkb > pre) asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x) : "memory");
      asm volatile("griddepcontrol.wait;" ::: "memory");
      trace_min(p.trace, 1);
      // (slot and parity are counted along: a division by the runtime ring depth per stage is felt)
      int sl = 0;
      uint32_t par = 0;
      for (int i = pre; i < nkb; ++i) {
        const uint32_t full = bars + 8 * sl;
        const uint32_t a = base + sl * stage_bytes;
        const int k = (kb0 + i) * BK;
        // (the epilogue warps fetch the activations of the first `pre` blocks)
        if (!mbar_wait(bars + 8 * (STAGES + sl), par, cta_abort, p.err)) break;
        mbar_expect_tx(full, wbytes);
        tma_load_2d(a, &map_w, k, n0, full);
        if (p.dual) tma_load_2d(a + A_BYTES, &map_w, k, p.up_off + n0, full);
        mbar_expect_tx(full, X_TILE);
        tma_load_2d(a + wbytes, &map_x, k, 0, full);
        if (++sl == STAGES) { sl = 0; par ^= 1u; }
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && nkb > 0) {
      const uint32_t idesc = umma_idesc(TN);
      // descriptors of slot 0: a slot or 16 k further on only the address field moves
      const uint64_t da0 = umma_desc(base), db0 = umma_desc(base + wbytes);
      const uint64_t dslot = stage_bytes >> 4;
      constexpr uint64_t DK = UMMA_K * 2 >> 4, DUP = A_BYTES >> 4;
      uint64_t off = 0;
      int sl = 0;
      uint32_t par = 0;
      bool ok = true;
      for (int i = 0; i < nkb; ++i) {
        ok = mbar_wait(bars + 8 * sl, par, cta_abort, p.err);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t da = da0 + off, db = db0 + off;
        umma_bf16(tmem_acc, da, db, idesc, i > 0 ? 1u : 0u);
#pragma unroll
        for (int kk = 1; kk < BK / UMMA_K; ++kk) umma_bf16_acc(tmem_acc, da + kk * DK, db + kk * DK, idesc);
        if (p.dual) {
          umma_bf16(tmem_acc + TN, da + DUP, db, idesc, i > 0 ? 1u : 0u);
#pragma unroll
          for (int kk = 1; kk < BK / UMMA_K; ++kk) umma_bf16_acc(tmem_acc + TN, da + DUP + kk * DK, db + kk * DK, idesc);
        }
        if (i + STAGES < nkb) umma_commit(bars + 8 * (STAGES + sl));  // (nobody waits for a slot's last use)
        off += dslot;
        if (++sl == STAGES) { sl = 0; par ^= 1u; off = 0; }
      }
      if (ok) umma_commit(bar_accum);
    }
  } else {
    // outputs (and the residual) belong to the stream order: wait for the preceding kernel
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int et = tid - 64;
    // The activations of the k blocks whose weights are already on their way: plain 16-byte loads by
    // these idle warps, stored in the 128-byte swizzle the MMA reads.  They are all there is between
    // the predecessor's end and the MMAs, and a TMA load takes about 0.4 us longer to come back.
    const int npre = min(nkb, STAGES);
    const int lg_rows = p.x_rows == 8 ? 3 : p.x_rows == 16 ? 4 : 5;
    const int chunks = npre << (lg_rows + 3);
    uint4 xv[XCH];
    load_x_chunks(p, kb0, et, chunks, lg_rows, xv);
    // The sums of squares of the norm that is handed over are asked for together with them: per token the producer's
    // per-CTA partials, 128 / G threads over the parts for each group of four tokens.
    const int lg_q = p.M <= 4 ? 0 : p.M <= 8 ? 1 : p.M <= 16 ? 2 : 3;
    const float* src = p.ss_in + ((et & ((1 << lg_q) - 1)) << 2) + (int64_t)(et >> lg_q) * 32;
    float4 ssv[SS_FIRST];
    if (p.ss_in) {
#pragma unroll
      for (int i = 0; i < SS_FIRST; ++i) {
        ssv[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if ((et >> lg_q) + i * (128 >> lg_q) < p.ss_parts) ssv[i] = __ldcg((const float4*)(src + (int64_t)i * (128 >> lg_q) * 32));
      }
    }
    if (p.splits > 1 && p.out_mode == 2) {
      // split-K: the elements this thread will finish first are known now; fetch their residuals (and
      // the next norm's gain) while the MMAs run instead of after the reduction
      const int lg = p.lg_rows_per, col = et >> lg;
      const int n = n0 + (split << lg) + (et & ((1 << lg) - 1));
      if (n < p.N) {
        if (col < p.M) asm volatile("ld.global.f32 %0, [%1];" : "=f"(res0) : "l"(p.residual + (int64_t)col * p.ldo + n) : "memory");
        if (col + (128 >> lg) < p.M)
          asm volatile("ld.global.f32 %0, [%1];" : "=f"(res1) : "l"(p.residual + (int64_t)(col + (128 >> lg)) * p.ldo + n) : "memory");
        if (p.xb_out) asm volatile("ld.global.f32 %0, [%1];" : "=f"(gain) : "l"(p.g_next + n) : "memory");
      }
    }
    store_x_chunks(base + wbytes, stage_bytes, et, chunks, lg_rows, xv);
    for (int c0 = et + 128 * XCH; c0 < chunks + et; c0 += 128 * XCH) {
      load_x_chunks(p, kb0, c0, chunks, lg_rows, xv);
      store_x_chunks(base + wbytes, stage_bytes, c0, chunks, lg_rows, xv);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("bar.sync 1, 128;" ::: "memory");
    if (et < npre) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bars + 8 * et) : "memory");
    if (p.ss_in) {
      // in a fixed order: a thread's parts, then a shuffle tree, then the four warps in order
      const int lg = lg_q;
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < SS_FIRST; ++i) { a.x += ssv[i].x; a.y += ssv[i].y; a.z += ssv[i].z; a.w += ssv[i].w; }
#pragma unroll 4
      for (int i = (et >> lg) + SS_FIRST * (128 >> lg); i < p.ss_parts; i += 128 >> lg) {
        const float4 v = __ldcg((const float4*)(src + (int64_t)(i - (et >> lg)) * 32));
        a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
      }
      for (int o = 16; o >= (1 << lg); o >>= 1) {
        a.x += __shfl_xor_sync(0xffffffffu, a.x, o);
        a.y += __shfl_xor_sync(0xffffffffu, a.y, o);
        a.z += __shfl_xor_sync(0xffffffffu, a.z, o);
        a.w += __shfl_xor_sync(0xffffffffu, a.w, o);
      }
      if (lane < (1 << lg)) *(float4*)(sc + 32 + (warp - 2) * 32 + lane * 4) = a;
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (et < p.M)
        sc[et] = 1.0f / sqrtf((((sc[32 + et] + sc[64 + et]) + sc[96 + et]) + sc[128 + et]) * p.ss_inv_h + p.ss_eps);
      asm volatile("bar.sync 1, 128;" ::: "memory");
    }
    // (the peers' barriers: waited for here, where there is time)
    if (cluster && !p.xstage_in_ring) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (nkb > 0) {
      acc_ok = mbar_wait(bar_accum, 0, cta_abort, p.err);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (tid == 64) trace_max(p.trace, 2);
    }
  }

  // the reduction this kernel contributes to: one more than the last one this rank pushed
  // (stable until this kernel's last CTA has seen every other CTA finish)
  uint32_t parity = 0;
  if (p.out_mode == 3 && warp >= 2) parity = peer_push_parity(p.push);
  if (cluster) {
    // (exchange area in the ring: every thread of every CTA of the cluster arrives only after its CTA's
    // loads have landed and its MMAs have read them; after this the rings may be written by the peers)
    __syncwarp();
    if (p.xstage_in_ring) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    if (p.xstage_in_ring || warp < 2) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  // with split-K a CTA whose accumulator never came pushes all the same: its peers count on the bytes
  // (the error word is set: what a peer makes of them is not a result)
  if (warp >= 2 && (acc_ok || cluster)) {
    const int q = warp & 3;
    const int row = q * 32 + lane;
    const int n = n0 + row;
    // split-K: every value goes straight into the exchange area of the CTA that finishes its row
    // (rows [r * 128 / S, (r + 1) * 128 / S) belong to cluster rank r), slot [this split][col][row]
    const int lg = p.lg_rows_per;
    const int xcols = (p.dual ? 2 : 1) * p.xstage_cols;
    uint32_t xdst = 0, xbar = 0;
    if (cluster) {
      const uint32_t owner = (uint32_t)(row >> lg);
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(xdst) : "r"(base + xoff), "r"(owner));
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(xbar) : "r"(bar_x), "r"(owner));
      xdst += (uint32_t)(((split * xcols) << lg) + (row & ((1 << lg) - 1))) * 4u;
    }
    if (cluster) {
#pragma unroll 1
      for (int c0 = 0; c0 < TN; c0 += 16) {
        if (c0 >= p.M) break;
        uint32_t g[16], u[16];
        tmem_ld16(tmem_acc + ((uint32_t)(q * 32) << 16) + (uint32_t)c0, g);
        if (p.dual) tmem_ld16(tmem_acc + ((uint32_t)(q * 32) << 16) + (uint32_t)(TN + c0), u);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          if (c0 + j >= p.M) break;
          st_async(xdst + ((uint32_t)(c0 + j) << (lg + 2)), g[j], xbar);
          if (p.dual) st_async(xdst + ((uint32_t)(p.xstage_cols + c0 + j) << (lg + 2)), u[j], xbar);
        }
      }
    } else {
      with_form(p, [&](auto form) {
        constexpr int FORM = decltype(form)::value;
        const bool in = n < p.N;
        float gn = 0.f;
        if (FORM == FORM_NORM && in) gn = p.g_plus_one ? 1.f + p.g_next[n] : p.g_next[n];
#pragma unroll 1
        for (int c0 = 0; c0 < TN; c0 += 16) {
          if (c0 >= p.M) break;
          uint32_t g[16], u[16];
          tmem_ld16(tmem_acc + ((uint32_t)(q * 32) << 16) + (uint32_t)c0, g);
          if (FORM == FORM_DUAL) tmem_ld16(tmem_acc + ((uint32_t)(q * 32) << 16) + (uint32_t)(TN + c0), u);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          int64_t o = (int64_t)c0 * p.ldo + n;
#pragma unroll
          for (int j = 0; j < 16; ++j, o += p.ldo) {
            if (c0 + j >= p.M) break;
            float r2 = 0.f;
            if (in)
              r2 = finish<FORM>(p, c0 + j, n, o, __uint_as_float(g[j]), FORM == FORM_DUAL ? __uint_as_float(u[j]) : 0.f, parity, sc,
                                FORM == FORM_NORM || FORM == FORM_RESIDUAL ? p.residual[o] : 0.f, gn);
            if (FORM == FORM_NORM) {
              // one CTA per tile here: the tile's 128 rows are summed per token, warp tree then warps in order
              for (int i = 16; i; i >>= 1) r2 += __shfl_xor_sync(0xffffffffu, r2, i);
              if (lane == 0) sq[q * 32 + c0 + j] = r2;
            }
          }
        }
      });
    }
  }
  if (warp >= 2 && p.ss_out && !cluster) {
    // (outside the branch above: all four epilogue warps must reach this barrier)
    asm volatile("bar.sync 2, 128;" ::: "memory");
    const int et = tid - 64;
    if (acc_ok && et < p.M) p.ss_out[(int64_t)blockIdx.x * 32 + et] = ((sq[et] + sq[32 + et]) + sq[64 + et]) + sq[96 + et];
  }

  if (warp >= 2 && p.out_mode != 3) {
    // the accumulators have been read: warp 1 gives the TMEM back beside the rest of the epilogue
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    asm volatile("bar.arrive 3, 160;" ::: "memory");
  }
  if (cluster) {
    // Arrived when every CTA of the cluster has issued its pushes; waited for before this CTA leaves,
    // so that no push can find its target gone even where a wait has given up.
    __syncwarp();
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    // the bytes themselves are counted on this CTA's own barrier, which costs one way across the
    // cluster where a barrier over all threads costs a return trip
    if (warp >= 2) {
      const bool got = mbar_wait_cluster(bar_x, 0, cta_abort, p.err) && !*cta_abort;
      // A thread finishes one row n and every (128 >> lg)-th token: what depends on n is done once, the rest
      // moves on by constants.
      const int S = p.splits, lg = p.lg_rows_per, et = tid - 64;
      const int rl = et & ((1 << lg) - 1), dc = 128 >> lg, n = n0 + (split << lg) + rl;
      const int cols = min(TN, p.M), turns = (cols + dc - 1) / dc;  // (the same number of turns for every thread)
      const float* x0 = (const float*)(gen + xoff) + et;
      const int step = ((p.dual ? 2 : 1) * p.xstage_cols) << lg, up = p.xstage_cols << lg;
      if (p.g_plus_one) gain += 1.f;
      with_form(p, [&](auto form) {
        constexpr int FORM = decltype(form)::value;
        auto all = [&](auto ranks) {
          constexpr int R = decltype(ranks)::value;
          const float* x = x0;
          int col = et >> lg;
          int64_t o = (int64_t)col * p.ldo + n;
          const int64_t dn = (int64_t)dc * p.ldo;
          float res = res0, next = res1;
#pragma unroll 1
          for (int t = 0; t < turns; ++t, col += dc, o += dn, x += 128) {
            const bool in = got && col < cols && n < p.N;
            float r2 = 0.f, third = 0.f;
            if (in) {
              if ((FORM == FORM_NORM || FORM == FORM_RESIDUAL) && col + 2 * dc < cols) third = p.residual[o + 2 * dn];  // two turns ahead
              const float g = add_ranks<R>(x, step);
              const float u = FORM == FORM_DUAL ? add_ranks<R>(x + up, step) : 0.f;
              r2 = finish<FORM>(p, col, n, o, g, u, parity, sc, res, gain);
            }
            res = next;
            next = third;
            if (FORM == FORM_NORM) {
              if (lg <= 5) {
                // a token's rows are neighbouring lanes
                for (int i = 1 << lg >> 1; i; i >>= 1) r2 += __shfl_xor_sync(0xffffffffu, r2, i);
                if (got && col < cols && rl == 0) p.ss_out[((int64_t)blockIdx.x * S + split) * 32 + col] = r2;
              } else if (got && col < cols) {
                sq[et + 128 * t] = r2;
              }
            }
          }
        };
        if (S == 16) all(std::integral_constant<int, 16>{});
        else if (S == 8) all(std::integral_constant<int, 8>{});
        else if (S == 4) all(std::integral_constant<int, 4>{});
        else all(std::integral_constant<int, 2>{});
      });
      if (p.ss_out && lg > 5) {
        asm volatile("bar.sync 2, 128;" ::: "memory");
        if (got && et < min(TN, p.M)) {
          float a = 0.f;
          for (int i = 0; i < 1 << lg; ++i) a += sq[(et << lg) + i];
          p.ss_out[((int64_t)blockIdx.x * S + split) * 32 + et] = a;
        }
      }
    }
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (*cta_abort) mbar_drain(bar_x, 0, p.err);  // (issued is not arrived: what is still on its way, after a wait gave up)
  }

  if (p.out_mode == 3) {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
  }
  if (warp == 1) {
    __syncwarp();
    if (p.out_mode != 3) asm volatile("bar.sync 3, 160;" ::: "memory");
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_acc), "r"(ncols) : "memory");
  }
  // every thread's pushes precede the barrier above
  if (p.out_mode == 3 && tid == 0) peer_push_done(p.push, (unsigned)p.total_ctas);
  if (tid == 64) trace_max(p.trace, 3);
}

template <int TN, int OCC>
int launch_dec(cg_ctx* c, const CUtensorMap& mw, const CUtensorMap& mx, const DecArgs& a, dim3 grid, size_t smem) {
  static PerDeviceSize configured_on;
  size_t& configured = configured_on.at(c->core->device);
  if (smem > configured) {
    CG_CUDA(c, cudaFuncSetAttribute(k_gemm_dec<TN, OCC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    CG_CUDA(c, cudaFuncSetAttribute(k_gemm_dec<TN, OCC>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    configured = smem;
  }
  CG_CUDA(c, launch_kernel(c, k_gemm_dec<TN, OCC>, grid, dim3(192), smem, a.splits, mw, mx, a));
  CG_LAUNCHED(c);
  return CG_OK;
}

}  // namespace

bool gemm_dec_supported(int64_t M, int64_t K) { return M >= 1 && M <= 32 && K % 8 == 0; }

// split-K: a power of two up to 16 (one cluster; above 8 is the non-portable size this GPU
// supports), at most about three CTAs per SM in total, at least two k blocks per CTA
static int dec_splits(int64_t tiles, int kb_total) {
  // (caps of 300 / 222 / 160 CTAs were measured 0.5 / 9 / 13 % slower per decode step, 600 4 % slower)
  const int cap = 3 * 148;
  int splits = 1;
  while (splits < 16 && tiles * (splits * 2) <= cap && kb_total / (splits * 2) >= 2) splits *= 2;
  // an empty slice would break the cluster shape
  auto slices = [&](int s) { const int per = (kb_total + s - 1) / s; return (kb_total + per - 1) / per; };
  while (splits > 1 && slices(splits) != splits) splits /= 2;
  return splits;
}

int gemm_dec_ss_parts(int64_t N, int64_t K) {
  const int64_t tiles = (N + BM - 1) / BM;
  return (int)(tiles * dec_splits(tiles, (int)((K + BK - 1) / BK)));
}

int gemm_dec(cg_ctx* c, const DecGemm& g) {
  if (g.M <= 0 || g.N <= 0) return CG_OK;
  if (!gemm_dec_supported(g.M, g.K) || g.K <= 0 || g.ldw % 8 || g.ldx % 8 || ((uintptr_t)g.w % 16) || ((uintptr_t)g.x % 16))
    return fail(c, CG_ERR_UNSUPPORTED, "gemm_dec: unsupported shape or alignment");
  const int tn = g.M <= 16 ? 16 : 32;
  const int64_t tiles = (g.N + BM - 1) / BM;
  const int kb_total = (int)((g.K + BK - 1) / BK);
  const int splits = dec_splits(tiles, kb_total);
  const int kb_per = (kb_total + splits - 1) / splits;
  const size_t wbytes = g.dual ? 2 * A_BYTES : A_BYTES;
  // up to 8 tokens: an 8-row activation box (1 KB instead of 2 per k block), which is what lets a
  // fourth ring stage fit beside the exchange area at three CTAs per SM
  const int x_rows = g.M <= 8 ? 8 : tn;
  const size_t stage = wbytes + (size_t)x_rows * BK * 2;
  // about a third of an SM's shared memory per CTA, so the next GEMM's CTAs can be resident
  // (and prefetching their weights) while this one computes
  // (the paired gate/up GEMM carries two weight tiles per stage, so the same budget would
  // leave it only two stages: it gets three, at two CTAs per SM)
  // The split-K exchange area (written by the other CTAs of the cluster, so outside the ring)
  // comes out of the same budget: three CTAs per SM may use 75 KB each, two 113 KB each.
  const int xstage_cols = splits > 1 ? (int)std::min<int64_t>(tn, g.M) : 0;
  const bool x_in_ring = tn == 32;  // above 16 tokens a separate area would cost the ring a stage (measured: 3 % per step)
  const size_t xarea = (size_t)(g.dual ? 2 : 1) * xstage_cols * BM * 4;
  const size_t xbytes = x_in_ring ? 0 : xarea;
  // (with the 8-row box the MMA of the last stage reads 1 KB past its activation slot: keep that inside the allocation)
  const size_t fixed = 1024 + 16 * 8 + 64 + 5 * 128 + (x_rows < tn ? 1024 : 0);
  // (smaller budgets -- 57 or 43 KB, 78 KB for the pair -- were measured 2-5 % slower per step)
  const size_t budget = (g.dual ? 113 * 1024 : 75 * 1024) - fixed;
  int stages = (int)std::max<size_t>(2, (budget > xbytes ? budget - xbytes : 0) / stage);
  // The paired kernel: three stages leave room for two CTAs per SM and nothing else, so when its
  // CTAs fill nearly all of those slots it takes two stages, and the next kernel's CTAs fit beside it
  // and fetch their weights early (Gemma-2-2B shape, 288 CTAs: 2.40 -> 2.25 ms per step; the
  // Llama-3.2-1B shape, 256 CTAs, measured 1-2 % better with three).
  if (g.dual && tiles * splits > 7 * 148 / 4) stages = std::min(stages, 2);
  stages = std::min(stages, std::max(kb_per, 2));
  stages = std::min(stages, 8);
  // the squared-output staging of the norm hand-over lives in the ring
  while ((g.ss_out || x_in_ring) && (x_in_ring ? xarea : 0) + (g.ss_out ? (size_t)SQ_FLOATS * 4 : 0) > (size_t)stages * stage) ++stages;
  const size_t smem = (size_t)stages * stage + xbytes + fixed;

  CUtensorMap mw, mx;
  CG_TRY(make_map(c, &mw, g.w, g.w_rows, g.K, g.ldw, BM));
  CG_TRY(make_map(c, &mx, g.x, g.M, g.K, g.ldx, x_rows));
  DecArgs a;
  a.out = g.out; a.ldo = g.ldo; a.residual = g.residual; a.out_mode = g.out_mode;
  a.dual = g.dual; a.act = g.act; a.up_off = (int)g.N;
  a.M = (int)g.M; a.N = (int)g.N; a.K = (int)g.K;
  a.kb_total = kb_total; a.kb_per_split = kb_per; a.splits = splits; a.stages = stages;
  a.lg_rows_per = 0;
  while (BM >> (a.lg_rows_per + 1) >= splits) ++a.lg_rows_per;
  a.x_rows = x_rows;
  a.x = (const __nv_bfloat16*)g.x; a.ldx = g.ldx;
  a.xstage_cols = xstage_cols;
  a.xstage_in_ring = x_in_ring && splits > 1 ? 1 : 0;
  a.err = c->core->dev_err;
  a.trace = c->trace_on ? (int)(c->trace_next++ % TRACE_SLOTS) : -1;
  a.total_ctas = (int)(tiles * splits);
  a.xb_out = g.xb_out; a.g_next = g.g_next; a.g_plus_one = g.g_plus_one; a.ss_out = g.ss_out;
  a.ss_in = g.ss_in; a.ss_parts = g.ss_parts; a.ss_inv_h = g.ss_in ? 1.0f / (float)g.K : 0.f; a.ss_eps = g.ss_eps;
  if (g.xb_out && (g.out_mode != 2 || g.dual || !g.g_next || !g.ss_out || g.ldo != g.N))
    return fail(c, CG_ERR_INVALID, "gemm_dec: the norm hand-over needs the residual epilogue on a dense output");
  if (g.out_mode == 3) {
    if (!g.push || g.dual || g.M * g.ldo > g.push->max_elems)
      return fail(c, CG_ERR_INVALID, "gemm_dec: the pushed addend does not fit the exchange area");
    a.push = *g.push;
  } else {
    a.push = PeerPush{};
  }
  dim3 grid((unsigned)tiles, 1, (unsigned)splits);
  // (register bound for 4 CTAs per SM: 0.861 -> 0.836 ms per Llama-3.2-1B decode step against a
  // bound for 3; bounds for 5 and 6 measured the same as 4)
  if (tn == 16) return launch_dec<16, 4>(c, mw, mx, a, grid, smem);
  return launch_dec<32, 4>(c, mw, mx, a, grid, smem);
}

}  // namespace cg

using namespace cg;

extern "C" int32_t cg_trace_enable(cg_ctx* c, int32_t on) {
  if (!c) return CG_ERR_INVALID;
  c->trace_on = on != 0;
  c->trace_next = 0;
  if (on) {
    std::vector<unsigned long long> init((size_t)TRACE_SLOTS * 4);
    for (int i = 0; i < TRACE_SLOTS; ++i) {
      init[i * 4 + 0] = init[i * 4 + 1] = ~0ull;
      init[i * 4 + 2] = init[i * 4 + 3] = 0ull;
    }
    CG_CUDA(c, cudaStreamSynchronize(c->core->stream));
    CG_CUDA(c, cudaMemcpyToSymbol(g_trace, init.data(), init.size() * 8));
  }
  return CG_OK;
}

extern "C" int32_t cg_trace_read(cg_ctx* c, uint64_t* out, int32_t slots) {
  if (!c || !out || slots < 0 || slots > TRACE_SLOTS) return CG_ERR_INVALID;
  CG_CUDA(c, cudaStreamSynchronize(c->core->stream));
  CG_CUDA(c, cudaMemcpyFromSymbol(out, g_trace, (size_t)slots * 32));
  return CG_OK;
}
