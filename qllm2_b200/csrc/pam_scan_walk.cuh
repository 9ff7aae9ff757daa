// Forward scan of which no backward will read the states (bf16, d = 64, 1..4 states): a CTA takes a sequence and a head and WALKS
// over its chunks.  A chunk's tiles are loaded once; they give the state the next chunk starts from and the output, and the
// state stays with the CTA (one state in registers, several in two fp32 slots each, written and read by the same SM, so in L2).
//
// What bounds it: the chain of phases of a chunk (tiles, weighted planes, state sums, de-interleave, scores, masks, products, stores),
// 18 k clocks for one state and 45 k for three with two CTAs per SM (three: a quarter of it the sums' way out of the accumulators, 42 %
// of the issue slots taken).  The form it replaces, chunk sums -> carry -> outputs as three passes over all chunks, ran three such chains, read
// k and v twice and moved every chunk's state (K * 32 KB for 48-96 KB of tokens and output) through HBM two to four times.  32 documents
// of 512..16384 tokens, 16 heads, one state: 1853 -> 1295 us; 48 chat prompts of 32..1024, 12 heads, three states: 327 -> 239; 256 prompts
// of 70, 12 heads, three states: 339 -> 203.
// Code is kept short (rolled loops, 16 columns at a time): the first version, written out, was 216 KB for three states, spilled, and
// missed the instruction cache; its score epilogue took 8.8 k clocks instead of 1.9 k.
//
// CTAs stay (two per SM) and draw sequences from a list ordered by length, longest first; the tiles of the next chunk, or of the next
// sequence's first, are requested as soon as the products have read this one's.
//
// A sequence that is long beside what the batch gives every SM to do would leave the chip to a few CTAs.  Its chunks are taken in the
// three passes instead (`split`): sums of every chunk by this kernel without its output part, the carry, and one-chunk jobs whose state
// is read from its slot, at the end of the same list.  Both ways give the same bits (the carry is the same sequence of fused multiply-adds).
// (One sequence of 60000 tokens among 32 of 100..300, 12 heads, as it is split / as kernels of their own for the three passes: one state
// 438 / 450 us, three 821 / 839.)
// Batches with few sequences and heads take the three passes as kernels of their own (scan_forward_only, pam_scan.cu).
#pragma once
#include "pam_scan_tc3.cuh"

namespace qpam {
namespace tcs {

// decays and factors of a step, 20 bytes a token and state: two sets, so that the next step's are formed while this one's output leaves
// (four states have room for one)
__host__ __device__ constexpr int walk_sets(int K) { return K <= 3 ? 2 : 1; }
__host__ __device__ constexpr size_t walk_smem(int K, bool out) { return 1024 + (out ? 3 : 2) * 32768 + (size_t)walk_sets(K) * K * TC * 20 + 512; }
// Both forms are built and launched for two CTAs per SM.  (The sums were built for three, of which two fitted for K = 2 and 3: 80 registers,
// 196 bytes spilled, eight columns at a time, and a third of the grid began behind the others' last jobs.  60000 tokens among 32 short
// sequences, 12 heads, all of them split: one state 501 -> 460 us, three 948 -> 865.)
constexpr int WALK_PER_SM = 2;
constexpr size_t SM_SMEM = 228 * 1024, CTA_RESERVED = 1024;
template <int K>
constexpr bool walk_fits() { return WALK_PER_SM * (walk_smem(K, true) + CTA_RESERVED) <= SM_SMEM && WALK_PER_SM * (walk_smem(K, false) + CTA_RESERVED) <= SM_SMEM; }
static_assert(walk_fits<1>() && walk_fits<2>() && walk_fits<3>() && walk_fits<KMAX>(), "CTAs per SM of the walking kernels");
// ScanParams::ticket: [0] next job of the outputs  [1] of the sums  [2] entries of the list  [3] how many of them, at its end, are chunks of split
// sequences: the jobs of the sums  [4] any sequence for the carry  [5] sequences of more chunks are split
enum { WT_OUT = 0, WT_SUM = 1, WT_JOBS = 2, WT_SPLIT_JOBS = 3, WT_CARRY = 4, WT_SPLIT = 5 };
constexpr int WALK_BINS = 1024;        // sequences are counted by their chunks, the longest (1023 and more) together

// What a call takes if sequences of more than a given number of chunks are split, in the time of a chunk that is walked with two CTAs on
// every SM (10 us with one state, 26 with three).  walked, split: chunks of either kind; longest_walked, longest_split: chunks of the
// longest sequence of either kind; per_cta: heads over the CTAs that the chip holds.  The walks end with the longest of them (0.6 a chunk
// once it has its SM for itself) or with their share of the work; a split chunk costs 0.7 for its sums before anything else begins and 0.8
// for its output, a link of the carry 0.01, the two launches 1.
// The call takes the cheapest split.  Measured over 32 batches and 1..4 states against the best of splitting above 0 / 0.6 / .. / 1.5 / 2 / 3
// times a CTA's share / never, it is within 2 % of the best on average and within 10 % everywhere; a fixed factor is not: of 48 prompts
// around 300 tokens (log-normal, deviation 1.5), 12 heads, one state, a split above 1 / 1.5 / 3 times the share takes 213 / 230 / 350 us, of
// 28 of 512..16384 1200 / 986 / 1130.
__host__ __device__ inline float walk_cost(float walked, float split, float longest_walked, float longest_split, float per_cta) {
  const float shared = per_cta * (walked + split);
  const float t = fmaxf(0.6f * longest_walked + 0.4f * fminf(longest_walked, shared), per_cta * (walked + 0.8f * split));
  return split > 0.f ? t + 1.f + 0.7f * per_cta * split + 0.01f * longest_split : t;
}

struct WalkStep {
  int32_t valid, h, b, c, t0, len, walk, pad;      // the chunk: tokens [t0, t0 + len) of row b
  WalkJob job;
};

// the first chunk of an entry
template <bool OUT>
__device__ __forceinline__ void walk_first(const ScanParams& p, unsigned int t, WalkStep& s) {
  const WalkJob& j = s.job;
  s.valid = 1;
  s.h = (int)(t % (unsigned int)p.H);
  s.b = p.geom.cu_seqlens != nullptr ? 0 : j.seq;
  s.c = j.c0;
  s.walk = OUT && j.c1 - j.c0 == j.nc;
  s.t0 = j.a + j.c0 * TC;
  s.len = min(TC, j.e - s.t0);
}
// entry `seq` of a call whose sequences are equally long
__device__ __forceinline__ WalkJob walk_uniform_job(const ScanParams& p, int seq) {
  const int nc = p.geom.nc_uniform;
  return WalkJob{seq, 0, nc, nc, 0, p.T, seq * (nc + 1), pool_slot_of(p, seq)};
}
__device__ __forceinline__ void walk_request_entry(WalkJob* smem_dst, const WalkJob* src) {
#pragma unroll
  for (int i = 0; i < 2; ++i)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(umma::smem_u32(smem_dst) + 16 * i), "l"(reinterpret_cast<const char*>(src) + 16 * i) : "memory");
}

template <int K, bool OUT>
__global__ void __launch_bounds__(256, WALK_PER_SM) k_tc_walk(const __grid_constant__ ChunkMaps maps, ScanParams p) {
  using namespace umma;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* RB = smem;                  // k tile, its planes, carried-state planes, the output on its way out
  unsigned char* RC = RB + 32768;            // v tile, weighted planes of the sums, its planes
  unsigned char* RA = RC + 32768;            // (OUT) q tile, its planes
  float* factors = reinterpret_cast<float*>(OUT ? RA + 32768 : RA);
  uint64_t* bars = reinterpret_cast<uint64_t*>(factors + walk_sets(K) * K * TC * 5);  // [0] q, v (sums alone: k, v)  [1] k  [2] sums  [3] scores  [4] products  [5] state
  WalkStep* steps = reinterpret_cast<WalkStep*>(bars + 6);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(steps + 2);
  int* failed = reinterpret_cast<int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr bool MULTI = K > 1;
  const bool packed = p.geom.cu_seqlens != nullptr;
  pdl_wait();
  unsigned int entries = (unsigned int)p.geom.S;
  const WalkJob* jobs = p.jobs;
  if (packed) {
    entries = p.ticket[OUT ? WT_JOBS : WT_SPLIT_JOBS];
    if (entries == 0u) return;               // (the sums of a call without split sequences)
    if (!OUT) jobs += p.ticket[WT_JOBS] - entries;
  }
  const unsigned int total = entries * (unsigned int)p.H;

  auto request_tiles = [&](const WalkStep& s) {
    const int row0 = (s.b * p.H + s.h) * p.T + s.t0;
    mbar_arrive_expect_tx(&bars[0], 4 * 16384);
#pragma unroll
    for (int kb = 0; kb < 2; ++kb) {
      tma_load_2d(RC + kb * 16384, &maps.x2, &bars[0], kb * 64, row0);
      if (OUT) tma_load_2d(RA + kb * 16384, &maps.a1, &bars[0], kb * 64, row0);
      else tma_load_2d(RB + kb * 16384, &maps.b1, &bars[0], kb * 64, row0);      // (no output waits in its region)
    }
  };
  auto request_k = [&](const WalkStep& s) {
    const int row0 = (s.b * p.H + s.h) * p.T + s.t0;
    mbar_arrive_expect_tx(&bars[1], 2 * 16384);
#pragma unroll
    for (int kb = 0; kb < 2; ++kb) tma_load_2d(RB + kb * 16384, &maps.b1, &bars[1], kb * 64, row0);
  };
  // Decays, factors and read-out weights of a step.  Warp k + 1 has state k, a lane four tokens: requested a step ahead, and formed
  // before the step begins.
  float graw[4];
  float2 craw[4];
  auto request_weights = [&](const WalkStep& s) {
    if (!s.valid || warp < 1 || warp > K) return;
    const size_t at = gamma_base(p, warp - 1, s.b, s.h, s.t0);
    warp_cumsum128_load(graw, p.gamma + at, s.len, lane);
    if (MULTI && OUT) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        craw[i] = make_float2(1.f, 0.f);
        if (p.coef != nullptr && 4 * lane + i < s.len) craw[i] = __ldg(reinterpret_cast<const float2*>(p.coef + (at + 4 * lane + i) * 2));
      }
    }
  };
  auto form_factors = [&](const WalkStep& s, int set) {
    if (!s.valid || warp < 1 || warp > K) return;
    float* Acum = factors + (set * K * 5 + warp - 1) * TC;           // [K][128] cumulative log-decay, then
    warp_cumsum128_finish(Acum, graw, s.len, p.eps, lane);
    __syncwarp();
    const float4 a4 = reinterpret_cast<const float4*>(Acum)[lane];
    const float a[4] = {a4.x, a4.y, a4.z, a4.w}, a_mid = Acum[TC / 2 - 1], a_last = Acum[TC - 1];
    const bool strong = a_last < STRONG_DECAY;
    float w[4], cf[4], rf[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      w[i] = __expf(fminf(0.f, a_last - a[i]));
      cf[i] = strong ? 1.f : __expf(a_mid - a[i]);
      rf[i] = p.q_scale * (strong ? 1.f : __expf(a[i] - a_mid));
    }
    reinterpret_cast<float4*>(Acum + 2 * K * TC)[lane] = make_float4(w[0], w[1], w[2], w[3]);      // [K][128] weights of the sums, e^{A_last - A_s}
    if (OUT) {
      reinterpret_cast<float4*>(Acum + K * TC)[lane] = make_float4(cf[0], cf[1], cf[2], cf[3]);    // [K][128] e^{A_m - A_s}
      float2* rho = reinterpret_cast<float2*>(factors + (set * K * 5 + 3 * K) * TC) + (warp - 1) * TC + 4 * lane;
#pragma unroll
      for (int i = 0; i < 4; ++i) rho[i] = MULTI ? make_float2(craw[i].x * rf[i], craw[i].y * rf[i]) : make_float2(rf[i], 0.f);      // c_k scale e^{A_t - A_m}
    }
  };

  if (tid == 0) {
    *failed = device_error_now();
#pragma unroll
    for (int i = 0; i < 6; ++i) mbar_init(&bars[i], 1);
    fence_barrier_init();
    const unsigned int t = blockIdx.x;       // (the counters start behind the grid)
    steps[0].valid = 0;
    if (t < total && *failed == 0) {
      steps[0].job = packed ? jobs[t / (unsigned int)p.H] : walk_uniform_job(p, (int)(t / (unsigned int)p.H));
      walk_first<OUT>(p, t, steps[0]);
      request_tiles(steps[0]);
    }
  }
  __syncwarp();
  if (warp == 0) tmem_alloc<OUT ? 256 : 128>(tmem_slot);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (OUT) pdl_trigger();                    // (the sums: by their end, see k_walk_carry)
  const uint32_t tmem = *tmem_slot;
  // thread 0: the entry to walk after the current one, drawn when the current one's last chunk is the next step (equally long
  // sequences: every gridDim.x-th entry)
  unsigned int ticket = blockIdx.x;
  auto draw = [&](const WalkStep& s) {
    if (s.c + 1 != s.job.c1) return;
    ticket += gridDim.x;
    if (packed) asm volatile("atom.global.add.u32 %0, [%1], 1;" : "=r"(ticket) : "l"(p.ticket + (OUT ? WT_OUT : WT_SUM)) : "memory");
  };
  if (tid == 0 && steps[0].valid) draw(steps[0]);
  const int q4 = warp & 3, hf = warp >> 2;
  const int r = q4 * 32 + lane;              // this thread's row (TMEM lane)
  const uint32_t tl = tmem + ((uint32_t)(q4 * 32) << 16);
  const uint32_t a_r = smem_u32(RA), b_r = smem_u32(RB), x_r = smem_u32(RC);
  const bool even = (lane & 1) == 0;
  const float sign = even ? 1.f : -1.f;      // Re U = D1[2j] + D2[2j+1], Im U = D2[2j] - D1[2j+1]
  uint32_t ph_sum = 0, ph_tile = 0, ph_out = 0, ph_state = 0;
  int cur = 0;
  request_weights(steps[0]);
  form_factors(steps[0], 0);
  __syncthreads();
  // One state: it stays in registers, column r of rows [32 hf, 32 hf + 32) (as the sums leave the accumulators).  (In slots, as K
  // states do it, 32 stores, 32 loads and a copy into shared memory a step: 22 k clocks instead of 18.)
  constexpr bool HELD = OUT && !MULTI;
  float S[HELD ? 32 : 1];

#pragma unroll 1
  while (steps[cur].valid) {
    const WalkStep& s = steps[cur];
    WalkStep& nx = steps[cur ^ 1];
    const bool job_ends = s.c + 1 == s.job.c1;
    // the job after this one: its ticket was drawn a step ago, its entry is requested here and looked at behind the sums
    const bool more = tid == 0 && job_ends && ticket < total;
    if (more && packed) walk_request_entry(&nx.job, jobs + ticket / (unsigned int)p.H);
    const float* Acum = factors + (walk_sets(K) == 2 ? cur : 0) * K * 5 * TC;
    const float *cfac = Acum + K * TC, *wrow = cfac + K * TC;
    const float2* rho = reinterpret_cast<const float2*>(wrow + K * TC);
    uint32_t strong_mask = 0;
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (Acum[k * TC + TC - 1] < STRONG_DECAY) strong_mask |= 1u << k;
    // where this chunk's states come from and go to
    const bool to_final = s.walk && s.c + 1 == s.job.nc;
    const bool sums = !OUT || (s.walk && (!to_final || p.s_final != nullptr || p.pool != nullptr));
    const int64_t from_slot = s.job.slot0 + (s.walk ? 1 + ((s.c - 1) & 1) : s.c);           // walking: slots 1 and 2 of the sequence in turn
    const int64_t to_slot = s.job.slot0 + (s.walk ? 1 + (s.c & 1) : s.c + 1);
    const bool has_state = OUT && (s.c > 0 || p.s0 != nullptr);
    auto entering = [&](int k) {
      return s.c == 0 ? p.s0 + (((size_t)k * p.geom.S + s.job.seq) * p.H + s.h) * (size_t)(TD * TD) * 2
                      : reinterpret_cast<const float*>(p.states + state_base(p, k, s.h, from_slot, TD));
    };
    if constexpr (HELD) {
      if (s.c == s.job.c0) {                 // a job begins: the state that enters its first chunk
        const float* prev = has_state ? entering(0) + hf * 4096 + r : nullptr;
#pragma unroll
        for (int i = 0; i < 32; ++i) S[i] = prev ? __ldcg(prev + i * 128) : 0.f;
      }
    }
    bool ok = mbar_wait(&bars[0], ph_tile, 241);
    // this thread's 16-byte pieces of the value tile (rows past the chunk's end: zeros, which also cancel whatever the key tile
    // holds in those rows), as in k_tc_chunk_outer
    const int row0_ = tid >> 4, c16 = tid & 15;
    const unsigned char* src = RC + (c16 >> 3) * 16384 + sw128(row0_, c16 & 7);
    unsigned char* planes = RC + sw128(row0_, c16 >> 1) + (c16 & 1) * 8;
    uint4 vxa[8];
#pragma unroll
    for (int it = 0; it < 8; ++it) {
      vxa[it] = make_uint4(0, 0, 0, 0);
      if (row0_ + 16 * it < s.len) vxa[it] = *reinterpret_cast<const uint4*>(src + 2048 * it);
    }
    if (OUT && lane == 0) tma_store_wait_read();        // the previous step's output has left the k region
    const int drow = tid & 127, dhb = tid >> 7;         // (a quarter-warp reads eight rows of one block: no bank conflict)
    if constexpr (OUT) {
      uint4 x[8];
      deint_read(RA, drow, dhb, x);
      __syncthreads();
      if (tid == 0) request_k(s);
      deint_write(RA, drow, dhb, x);
    } else {
      __syncthreads();
    }
    // the entering state as words of its bf16 planes, times the chunk constant (two columns a word: a lane takes row i or i + 2 for itself
    // and the lane two further on); they go to the k region once the scores have been formed
    uint32_t sw[HELD ? 16 : 1];
    if constexpr (HELD) {
      const float cst = state_const(Acum, strong_mask, 0);
      const bool upper = lane & 2;
#pragma unroll
      for (int m = 0; m < 16; ++m) {
        const int i = (m >> 1) * 4 + (m & 1);
        const float mine = upper ? S[i + 2] : S[i], got = __shfl_xor_sync(0xffffffffu, upper ? S[i] : S[i + 2], 2);
        sw[m] = upper ? pack_bf162(cst * got, cst * mine) : pack_bf162(cst * mine, cst * got);
      }
    }
    if (sums) {
      constexpr int G = 16;                    // columns at a time
      float pv[G];                             // that many of the thread's elements of the entering state, ahead of their use
      // the sums of state k leave the accumulators: S' = g S + U, U as in k_tc_chunk_outer
      auto sums_out = [&](int k) {
        if constexpr (HELD) {
          const float g = __expf(Acum[TC - 1]);
#pragma unroll
          for (int hh = 0; hh < 4; ++hh) {
            float d1[8], d2[8];
            tmem_ld8x2(tl + hf * 32 + hh * 8, d1, tl + 64 + hf * 32 + hh * 8, d2);
#pragma unroll
            for (int i = 0; i < 8; i += 2) {
              const float2 o = make_float2(__shfl_xor_sync(0xffffffffu, d2[i], 1), __shfl_xor_sync(0xffffffffu, d2[i + 1], 1));
              const float2 u = ffma2(make_float2(g, g), make_float2(S[hh * 8 + i], S[hh * 8 + i + 1]), ffma2(make_float2(sign, sign), make_float2(d1[i], d1[i + 1]), o));
              S[hh * 8 + i] = u.x;
              S[hh * 8 + i + 1] = u.y;
            }
          }
          if (to_final) {
            FinalDest fin;
            fin.init(p, s.job.seq, s.job.pool_slot, 0, s.h);
            fin.store(p, hf * 4096 + r, S, even, ok);
          }
          return;
        }
        const uint32_t from = tl + (OUT ? (uint32_t)(k & 1) * 128u : 0u);
        // lane n' = 2j+c holds column i, state[i][j][c] at i*128 + n'
        const float g = __expf(Acum[k * TC + TC - 1]);
        const float* prev = has_state ? entering(k) + hf * 4096 + r : nullptr;
        float* next = reinterpret_cast<float*>(p.states + state_base(p, k, s.h, to_slot, TD)) + hf * 4096 + r;
        FinalDest fin;
        if (to_final) fin.init(p, s.job.seq, s.job.pool_slot, k, s.h);
#pragma unroll 1
        for (int hh = 0; hh < 32 / G; ++hh) {
          float d1[G], d2[G];
          const uint32_t col = (uint32_t)(hf * 32 + hh * G);
          tmem_ld16x2(from + col, d1, from + 64 + col, d2);
#pragma unroll
          for (int i = 0; i < G; i += 2) {      // two columns an instruction
            const float2 o = make_float2(__shfl_xor_sync(0xffffffffu, d2[i], 1), __shfl_xor_sync(0xffffffffu, d2[i + 1], 1));
            float2 u = ffma2(make_float2(sign, sign), make_float2(d1[i], d1[i + 1]), o);
            if (has_state) u = ffma2(make_float2(g, g), make_float2(pv[i], pv[i + 1]), u);
            d1[i] = u.x;
            d1[i + 1] = u.y;
          }
          if (has_state) {
            if (OUT && hh == 0) {
#pragma unroll
              for (int i = 0; i < G; ++i) pv[i] = __ldcg(prev + 2048 + i * 128);
            }
          }
          if (to_final) {
            fin.store(p, (int)col * 128 + r, d1, even, ok);
          } else if (ok) {
#pragma unroll
            for (int i = 0; i < G; ++i) next[i * 128] = d1[i];
            next += 128 * G;
          }
        }
        if (!OUT && ok && tid == 0) p.chunk_decay[((size_t)k * p.H + s.h) * p.nslots + s.job.slot0 + s.c + 1] = g;
      };
#pragma unroll 1
      for (int k = 0; k <= K; ++k) {
        if (!OUT && k > 0) sums_out(k - 1);
        if (k < K) {
#pragma unroll
          for (int it = 0; it < 8; ++it) {
            const float w = wrow[k * TC + row0_ + 16 * it];
            const uint32_t vw[4] = {vxa[it].x, vxa[it].y, vxa[it].z, vxa[it].w};
            float2 x[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) x[e] = fmul2(unpack_bf162(vw[e]), make_float2(w, w));
            *reinterpret_cast<uint2*>(planes + 2048 * it) = make_uint2(pack_bf162(x[0].x, x[1].x), pack_bf162(x[2].x, x[3].x));
            *reinterpret_cast<uint2*>(planes + 16384 + 2048 * it) = make_uint2(pack_bf162(x[0].y, x[1].y), pack_bf162(x[2].y, x[3].y));
          }
          fence_proxy_async();
          tc_fence_before();
          __syncthreads();
          if (warp == 0 && elect_one()) {
            tc_fence_after();
            if (OUT && k == 0) mbar_wait(&bars[1], ph_tile, 243);
            const uint32_t d = tmem + (OUT ? (uint32_t)(k & 1) * 128u : 0u);
            constexpr uint32_t idesc = idesc_bf16(128, 64, true, true);
            mma_run(d, smem_desc_sw128(b_r, 16384, 1024), smem_desc_sw128(x_r, 16, 1024), 128, 128, idesc, 8, false);      // D1 = k'^T (w Re v)
            mma_run(d + 64, smem_desc_sw128(b_r, 16384, 1024), smem_desc_sw128(x_r + 16384, 16, 1024), 128, 128, idesc, 8, false);      // D2 = k'^T (w Im v)
            mma_commit(&bars[2]);
          }
          __syncwarp();
        }
        if (OUT && k > 0) sums_out(k - 1);      // (beside this state's products: they go to the other half of the accumulators)
        if (k == K) break;
        if (MULTI && has_state) {
          const float* prev = entering(k) + hf * 4096 + r;
#pragma unroll
          for (int i = 0; i < G; ++i) pv[i] = __ldcg(prev + i * 128);
        }
        ok = mbar_wait(&bars[2], ph_sum, 242) && ok;
        ph_sum ^= 1;
        tc_fence_after();
      }
    }
    if (tid == 0) {                          // the step after this one (known to all behind the next barrier)
      if (!job_ends) {
        nx = s;
        nx.c = s.c + 1;
        nx.t0 = s.t0 + TC;
        nx.len = min(TC, s.job.e - nx.t0);
      } else {
        nx.valid = 0;
        if (more) {
          if (packed) asm volatile("cp.async.wait_all;" ::: "memory");
          else nx.job = walk_uniform_job(p, (int)(ticket / (unsigned int)p.H));
          walk_first<OUT>(p, ticket, nx);
        }
      }
      if (nx.valid) draw(nx);
    }
    if constexpr (OUT) {
      // ---- the planes of v, exact, and of k
#pragma unroll
      for (int it = 0; it < 8; ++it) {
        const uint4 v = vxa[it];
        *reinterpret_cast<uint2*>(planes + 2048 * it) = make_uint2(__byte_perm(v.x, v.y, 0x5410), __byte_perm(v.z, v.w, 0x5410));
        *reinterpret_cast<uint2*>(planes + 16384 + 2048 * it) = make_uint2(__byte_perm(v.x, v.y, 0x7632), __byte_perm(v.z, v.w, 0x7632));
      }
      ok = mbar_wait(&bars[1], ph_tile, 243) && ok;
      {
        uint4 x[8];
        deint_read(RB, drow, dhb, x);
        tc_fence_before();                   // (the sums have left the accumulators)
        __syncthreads();
        deint_write(RB, drow, dhb, x);
      }
      fence_proxy_async();
      __syncthreads();
      if (warp == 0 && elect_one()) {
        tc_fence_after();
        bw_issue_scores(tmem, a_r, b_r);
        mma_commit(&bars[3]);
      }
      __syncwarp();
      request_weights(nx);
      ok = mbar_wait(&bars[3], ph_out, 244) && ok;
      tc_fence_after();
      if constexpr (!MULTI) {
        // one state: as chunk_job<M_FWD>
        const bool strong = strong_mask != 0;
        if (has_state) {
          unsigned char* plane = RB + (lane & 1) * 8192 + ((r >> 2) & 3) * 4;      // columns j0 = 2 (r / 4) and j0 + 1 of plane re or im
#pragma unroll
          for (int m = 0; m < 16; ++m) *reinterpret_cast<uint32_t*>(plane + sw128(hf * 32 + (m >> 1) * 4 + (m & 1) + (lane & 2), r >> 4)) = sw[m];
        }
        bw_epi_scores(true, tl, q4, hf, r, s.len, strong, cfac, Acum, p.q_scale, 1.f);
        tmem_st_wait();
        fence_proxy_async();
        tc_fence_before();
        __syncthreads();
        const bool two_step = strong && has_state;
        if (two_step) {                      // the carried-state product alone, then every row rescaled by its own decay
          if (warp == 0 && elect_one()) {
            tc_fence_after();
            bw_issue_state(false, tmem, a_r, b_r, false);
            mma_commit(&bars[5]);
          }
          __syncwarp();
          ok = mbar_wait(&bars[5], ph_state, 246) && ok;
          ph_state ^= 1;
          tc_fence_after();
          rescale_acc_half(tl, hf, p.q_scale * __expf(Acum[r]));
          tc_fence_before();
          __syncthreads();
        }
        if (warp == 0 && elect_one()) {
          tc_fence_after();
          const bool state_now = has_state && !strong;
          if (state_now) bw_issue_state(false, tmem, a_r, b_r, false);
          bw_issue_out(tmem, x_r, two_step || state_now);
          mma_commit(&bars[4]);
        }
        __syncwarp();
        if (walk_sets(K) == 2) form_factors(nx, cur ^ 1);
        ok = mbar_wait(&bars[4], ph_out, 247) && ok;
        tc_fence_after();
      } else {
        // K states: as k_tc_chunk_fwdK
        float2 rk[K];
#pragma unroll
        for (int k = 0; k < K; ++k) rk[k] = rho[k * TC + r];
        kstate_scores<K>(tl, q4, hf, r, strong_mask, rk, cfac, Acum);
        if (has_state) kstate_planes2(RB, entering(0), entering(1), state_const(Acum, strong_mask, 0), state_const(Acum, strong_mask, 1), tid);
        fence_proxy_async();
        tc_fence_before();
        __syncthreads();
        if (warp == 0 && elect_one()) {
          tc_fence_after();
          bw_issue_out(tmem, x_r);
          mma_commit(&bars[4]);
        }
        __syncwarp();
        if (walk_sets(K) == 2) form_factors(nx, cur ^ 1);
        ok = mbar_wait(&bars[4], ph_out, 247) && ok;
        tc_fence_after();
        if (has_state) {
#pragma unroll 1
          for (int pass = 0; pass * 2 < K; ++pass) {
            const int k_mine = pass * 2 + hf;
            if (pass > 0) {
#pragma unroll 1
              for (int k = pass * 2; k < K && k < pass * 2 + 2; ++k) kstate_planes(RB + (k & 1) * 16384, entering(k), state_const(Acum, strong_mask, k), tid);
            }
            if (k_mine < K) kstate_rows<K>(tl, RA, hf, r, k_mine, strong_mask, rk, Acum);
            fence_proxy_async();
            tc_fence_before();
            __syncthreads();
            if (warp == 0 && elect_one()) {
              tc_fence_after();
              kstate_issue(tmem, b_r, pass * 2 + 1 < K ? 2 : 1);
              mma_commit(&bars[5]);
            }
            __syncwarp();
            ok = mbar_wait(&bars[5], ph_state, 248) && ok;
            ph_state ^= 1;
            tc_fence_after();
          }
        }
      }
      // every product has read its operands: the next tiles may come
      if (tid == 0 && nx.valid) request_tiles(nx);
      // ---- the output leaves through the k region: 32 rows x 128 bytes a warp, one TMA store each; a ragged chunk (its rows past
      // the end belong to someone else) stores per lane
      const bool bulk = warp_agrees(ok) && s.len == TC;
      const float rf = MULTI || strong_mask != 0 ? 1.f : rho[r].x;
      __nv_bfloat16* orow = reinterpret_cast<__nv_bfloat16*>(p.y) + (p.y_token_major ? (((size_t)s.b * p.T + s.t0 + r) * p.H + s.h) * (size_t)(TD * 2)
                                                                                     : token_base(p, s.b, s.h, s.t0 + r, TD)) + hf * 64;
      unsigned char* wbox = RB + hf * 16384 + q4 * 4096;
      const uint4 none[4] = {};
#pragma unroll 1
      for (int cc = 0; cc < 2; ++cc)
        bw_epi_out<false>(false, tl, 2 * hf + cc, rf, orow + cc * 32, none, ok && r < s.len, bulk ? wbox + lane * 128 : nullptr, lane & 7);
      if (bulk) {
        fence_proxy_async();
        __syncwarp();
        if (lane == 0)
          tma_store_2d_keep(&maps.out, wbox, p.y_token_major ? s.h * 128 + hf * 64 : hf * 64,
                            (p.y_token_major ? s.b * p.T + s.t0 : (s.b * p.H + s.h) * p.T + s.t0) + q4 * 32);
      }
      ph_out ^= 1;
    } else {
      if (tid == 0 && nx.valid) request_tiles(nx);
    }
    ph_tile ^= 1;
    tc_fence_before();
    const bool all_ok = __syncthreads_and(ok);
    tc_fence_after();
    cur ^= 1;
    if (!all_ok) {                           // a wait gave up: no more work; the tiles on their way land first
      if (steps[cur].valid) mbar_wait(&bars[0], ph_tile, 249);
      break;
    }
    if (!OUT) request_weights(steps[cur]);
    if (!OUT || walk_sets(K) == 1) {
      form_factors(steps[cur], walk_sets(K) == 2 ? cur : 0);
      __syncthreads();
    }
  }
  if (lane == 0) tma_store_wait_read();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc<OUT ? 256 : 128>(tmem);
  }
}

// The list of a packed call, one CTA: chunks before every sequence (descriptor checked as in k_chunk_prefix_checked), which sequences are
// split (walk_cost), those to walk by falling length, then the chunks of the split ones.
__global__ void __launch_bounds__(1024) k_walk_plan(ScanParams p, int32_t* __restrict__ prefix, WalkJob* __restrict__ jobs, int ctas, int bad_code) {
  __shared__ int hist[WALK_BINS];            // sequences by their chunks, then where those of a length begin in the list
  __shared__ int wsum[32];
  __shared__ int carry_s, bad_s, special_s, split_s, longest_s;
  __shared__ unsigned long long best_s;
  pdl_wait();
  pdl_trigger();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, S = p.geom.S;
  const int32_t* cu = p.geom.cu_seqlens;
  hist[tid] = 0;
  if (tid == 0) {
    carry_s = special_s = split_s = longest_s = 0;
    best_s = ~0ull;
    bad_s = cu[0] != 0;
    prefix[0] = 0;
  }
  __syncthreads();
  // inclusive scan over the CTA; `all` is the total
  auto scan = [&](int n, int& all) {
    int inc = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    if (warp == 0) {
      int w = wsum[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += t;
      }
      wsum[lane] = w;
    }
    __syncthreads();
    if (warp > 0) inc += wsum[warp - 1];
    all = wsum[31];
    __syncthreads();
    return inc;
  };
  int first = 0, end = 0, slot = -1, before_me = 0;      // of sequence tid (all of a call's, if there are no more than threads)
  for (int base = 0; base < S; base += 1024) {
    const int s = base + tid;
    int n = 0;
    if (s < S) {
      const int a = cu[s], e = cu[s + 1];
      if (base == 0) {
        first = a;
        end = e;
        slot = pool_slot_of(p, s);
      }
      if (!(e >= a && e <= p.T)) bad_s = 1;
      n = (max(0, e - a) + TC - 1) / TC;
    }
    int all;
    const int inc = scan(n, all), before = carry_s;
    if (s < S) prefix[s + 1] = before + inc;
    if (base == 0) before_me = inc - n;
    __syncthreads();
    if (tid == 0) carry_s = before + all;
    __syncthreads();
  }
  const int C = carry_s;
  if (bad_s) {
    for (int s = tid; s <= S; s += 1024) prefix[s] = 0;
    if (tid == 0) {
      for (int i = 0; i < 6; ++i) p.ticket[i] = i == WT_CARRY ? 1u : 0u;      // (every sequence is empty now: its final state is its first)
      umma::record_device_error(bad_code);
    }
    return;
  }
  auto chunks_of = [&](int s) { return s < 1024 ? (end - first + TC - 1) / TC : prefix[s + 1] - prefix[s]; };
  int longest = 0;
  for (int s = tid; s < S; s += 1024) {
    const int nc = chunks_of(s);
    longest = max(longest, nc);
    if (nc > 0) atomicAdd(&hist[min(nc, WALK_BINS - 1)], 1);
    else special_s = 1;
  }
  longest = __reduce_max_sync(0xffffffffu, longest);
  if (lane == 0 && longest > 0) atomicMax(&longest_s, longest);
  __syncthreads();
  // thread x looks at a split above x chunks, where there are sequences of so many (x = 0: every one is split)
  longest = longest_s;
  const int count = hist[tid];
  int below_last;
  const int upto = scan(tid < WALK_BINS - 1 ? count * tid : 0, below_last);
  if (count > 0 || tid == 0) {
    const bool all = tid == WALK_BINS - 1;
    const int walked_chunks = all ? C : upto;
    const float t = walk_cost((float)walked_chunks, (float)(C - walked_chunks), (float)(all ? longest : tid), (float)longest, (float)p.H / (float)ctas);
    atomicMin(&best_s, (unsigned long long)__float_as_uint(t) << 32 | (unsigned int)(WALK_BINS - 1 - tid));      // (of equals the one that splits less)
  }
  __syncthreads();
  const int best = WALK_BINS - 1 - (int)(unsigned int)best_s, above = best == WALK_BINS - 1 ? 0x3fffffff : best;
  int walked;
  const int bin = WALK_BINS - 1 - tid, mine = bin <= above ? hist[bin] : 0, inc = scan(mine, walked);      // longest first
  hist[bin] = inc - mine;
  __syncthreads();
  for (int s = tid; s < S; s += 1024) {
    const int nc = chunks_of(s);
    if (nc > above) special_s = 1;
    else if (nc > 0)
      jobs[atomicAdd(&hist[min(nc, WALK_BINS - 1)], 1)] = s < 1024 ? WalkJob{s, 0, nc, nc, first, end, before_me + s, slot}
                                                                  : WalkJob{s, 0, nc, nc, cu[s], cu[s + 1], prefix[s] + s, pool_slot_of(p, s)};
  }
  __syncthreads();
  if (special_s)
    for (int x = tid; x < C; x += 1024) {
      int lo = 0, hi = S;                    // the last s with prefix[s] <= x
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (prefix[mid] <= x) lo = mid; else hi = mid;
      }
      const int nc = prefix[lo + 1] - prefix[lo];
      if (nc > above) {
        const int at = atomicAdd(&split_s, 1), c = x - prefix[lo];
        jobs[walked + at] = WalkJob{lo, c, c + 1, nc, cu[lo], cu[lo + 1], prefix[lo] + lo, pool_slot_of(p, lo)};
      }
    }
  __syncthreads();
  if (tid == 0) {
    p.ticket[WT_OUT] = (unsigned int)ctas;               // (behind the grids of the two: a CTA's first job is its index)
    p.ticket[WT_SUM] = (unsigned int)ctas;
    p.ticket[WT_JOBS] = (unsigned int)(walked + split_s);
    p.ticket[WT_SPLIT_JOBS] = (unsigned int)split_s;
    p.ticket[WT_CARRY] = (unsigned int)special_s;
    p.ticket[WT_SPLIT] = (unsigned int)above;
  }
}

// The carry of split sequences (of all of them where no list has been made), and the final states of empty ones:
// S_c+1 = g_c S_c + U_c, in place over the slots, as k_state_scan; the last state goes to its destination only, the first is written
// where it is given, and no slot at all where no output will read them (a call for final states alone).  CTAs take (sequence, head and
// state, eighth of a state) in turn: a grid with one for each took 78 us to find out that there was nothing to do (256 short prompts, 36
// heads and states).
// Where sums are formed before it, it is called by their end, not by their start: a long chain is only a few CTAs, and called early these
// piled up on the SMs that were free first (60000 tokens among 32 short sequences, 12 heads, one state: 547 -> 453 us; three, 893 -> 838).
__global__ void __launch_bounds__(256) k_walk_carry(ScanParams p) {
  pdl_wait();
  pdl_trigger();
  const bool packed = p.geom.cu_seqlens != nullptr;
  if (p.ticket != nullptr && p.ticket[WT_CARRY] == 0u) return;
  const int above = p.ticket != nullptr ? (int)p.ticket[WT_SPLIT] : 0;
  const bool keep = p.y != nullptr;
  constexpr int n4 = TD * TD / 2, UN = 4;
  const int64_t items = (int64_t)p.geom.S * p.H * p.K * (n4 / 256);
  for (int64_t it = blockIdx.x; it < items; it += gridDim.x) {
    const int64_t sh = it / (n4 / 256);
    const int seq = (int)(sh / (p.H * p.K)), hk = (int)(sh - (int64_t)seq * (p.H * p.K)), k = hk / p.H, h = hk - k * p.H;
    const int nc = packed ? p.geom.chunk_prefix[seq + 1] - p.geom.chunk_prefix[seq] : p.geom.nc_uniform;
    if ((nc > 0 && nc <= above) || (nc == 1 && p.finish == FIN_ONLY)) continue;
    const int64_t slot0 = packed ? (int64_t)p.geom.chunk_prefix[seq] + seq : (int64_t)seq * (nc + 1);
    const int e4 = (int)(it % (n4 / 256)) * 256 + threadIdx.x;
    float4* st = reinterpret_cast<float4*>(p.states + state_base(p, k, h, slot0, TD)) + e4;
    const float* dec = p.chunk_decay + ((size_t)k * p.H + h) * p.nslots + slot0;
    const size_t ext = ((((size_t)k * p.geom.S + seq) * p.H + h) * (size_t)(TD * TD)) / 2 + e4;
    float4 cur = p.s0 != nullptr ? reinterpret_cast<const float4*>(p.s0)[ext] : make_float4(0.f, 0.f, 0.f, 0.f);
    if (p.s0 != nullptr && keep) st[0] = cur;
    for (int c = 0; c < nc; c += UN) {
      float4 u[UN];
      float g[UN];
#pragma unroll
      for (int i = 0; i < UN; ++i)
        if (c + i < nc) {
          u[i] = st[(size_t)(c + i + 1) * n4];
          g[i] = dec[c + i + 1];
        }
#pragma unroll
      for (int i = 0; i < UN; ++i)
        if (c + i < nc) {
          if (c + i == 0 && p.s0 == nullptr) {
            cur = u[0];
            continue;
          }
          cur.x = fmaf(g[i], cur.x, u[i].x);
          cur.y = fmaf(g[i], cur.y, u[i].y);
          cur.z = fmaf(g[i], cur.z, u[i].z);
          cur.w = fmaf(g[i], cur.w, u[i].w);
          if (keep && c + i + 1 < nc) st[(size_t)(c + i + 1) * n4] = cur;
        }
    }
    if (p.s_final != nullptr) reinterpret_cast<float4*>(p.s_final)[ext] = cur;
    const int slot = pool_slot_of(p, seq);
    if (slot >= 0) store_final4(p, pool_block(p, slot, k, h, TD) + (int64_t)e4 * 4, cur);
  }
}

}  // namespace tcs
}  // namespace qpam
