// Tensor-core (tcgen05 / TMEM / TMA) kernels of the chunked PAM scan for bf16 token tensors,
// head dim 64, one state.  Chunks are 128 tokens, so every MMA is M = 128.
//
// This file: the chunk-local state sums (k_tc_chunk_outer).  The
// state sums run as real bf16 MMAs on the INTERLEAVED (re, im) rows as they sit in memory: a token
// row of 64 complex numbers is a 128-element real vector x = (r0, i0, r1, i1, ...); with
// cj(x) = (r0, -i0, ...) the real and imaginary parts of v (x) conj(k) come from the operand rows
// w cj(k), w (ki, kr) against the de-interleaved planes Re v, Im v.  The chunk outputs and
// gradients are in pam_scan_tc2.cuh.
#pragma once
#include "pam_scan_kernels.cuh"
#include "umma.cuh"

namespace qpam {
namespace tcs {

constexpr int TC = 128;   // tokens per chunk
constexpr int TD = 64;    // head dim (complex); a token row is 2*TD bf16 = 256 bytes

// byte offset of (row, 16-byte chunk c in 0..7) inside a [rows][128 B] block with the 128-byte swizzle
__device__ __forceinline__ uint32_t sw128(int row, int c) { return (uint32_t)row * 128u + (uint32_t)((c ^ (row & 7)) << 4); }

__device__ __forceinline__ float2 unpack_bf162(uint32_t w) {
  return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w));
}
__device__ __forceinline__ uint32_t pack_bf162(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// inclusive cumulative sum of log(gamma + eps) over 128 tokens by one warp (4 tokens per lane)
// (two halves, so that a caller can put other loads between the request for the decays and their first use)
__device__ __forceinline__ void warp_cumsum128_load(float (&g)[4], const float* __restrict__ gamma, int len, int lane) {
  const int t = 4 * lane;
#pragma unroll
  for (int i = 0; i < 4; ++i) g[i] = (t + i < len) ? __ldg(gamma + t + i) : 1.f;
}
__device__ __forceinline__ void warp_cumsum128_finish(float* A, const float (&g)[4], int len, float eps, int lane) {
  const int t = 4 * lane;
  float x[4];
  // log(gamma + eps) without the full-precision logf (~500 clocks of the chain that the first barrier of a chunk job
  // waits for).  Decays close to 1 are the ones whose errors would add up over thousands of tokens, so they get the
  // series of log1p(u), u = x - 1 (exact by Sterbenz for x in [0.5, 2]), to fp32 rounding: |u| < 1/16, six terms,
  // truncation < u^7/7 < 6e-10.  The rest takes the hardware logarithm (absolute error <= 2^-22 per token; such a
  // sequence has forgotten a token after a few hundred steps, long before those errors add up to 1e-4).  Every
  // tensor-core kernel forms its decays here, so chunk sums, carried states and outputs agree.
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float xg = g[i] + eps, u = xg - 1.f;
    const float series = u * fmaf(u, fmaf(u, fmaf(u, fmaf(u, fmaf(u, -1.f / 6.f, 0.2f), -0.25f), 1.f / 3.f), -0.5f), 1.f);
    x[i] = (t + i < len) ? (fabsf(u) < 0.0625f ? series : __logf(xg)) : 0.f;
  }
  x[1] += x[0];
  x[2] += x[1];
  x[3] += x[2];
  float incl = x[3];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float n = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += n;
  }
  const float excl = incl - x[3];
#pragma unroll
  for (int i = 0; i < 4; ++i) A[t + i] = excl + x[i];
}
__device__ __forceinline__ void warp_cumsum128(float* A, const float* __restrict__ gamma, int len, float eps, int lane) {
  float g[4];
  warp_cumsum128_load(g, gamma, len, lane);
  warp_cumsum128_finish(A, g, len, eps, lane);
}

// Where a sequence's final state goes: s_final and / or the sequence's pool slot.  A lane holds one column (n' = q4 * 32 + lane) of every row.
struct FinalDest {
  float* f;                 // s_final block, or null
  int64_t pool;             // first scalar of the pool block, or -1
  __device__ __forceinline__ void init(const ScanParams& p, int seq, int pool_slot, int k, int h) {
    f = p.s_final ? p.s_final + (((size_t)k * p.geom.S + seq) * p.H + h) * (size_t)(TD * TD) * 2 : nullptr;
    pool = pool_slot >= 0 ? pool_block(p, pool_slot, k, h, TD) : -1;
  }
  // rows i .. i + N - 1 of the lane's column; off: the scalar of row i
  template <int N>
  __device__ __forceinline__ void store(const ScanParams& p, int off, const float (&u)[N], bool even, bool ok) const {
    if (f && ok) {
#pragma unroll
      for (int i = 0; i < N; ++i) f[off + i * 2 * TD] = u[i];
    }
    if (pool < 0) return;
    if (p.pool_bf16) {           // the even lane of a pair takes both columns of row i, the odd lane those of row i + 1
      __nv_bfloat16* at = reinterpret_cast<__nv_bfloat16*>(p.pool) + pool + (even ? off : off - 1 + 2 * TD);
#pragma unroll
      for (int i = 0; i < N; i += 2) {
        const float x = __shfl_xor_sync(0xffffffffu, even ? u[i + 1] : u[i], 1);
        if (ok) *reinterpret_cast<uint32_t*>(at + i * 2 * TD) = even ? pack_bf162(u[i], x) : pack_bf162(x, u[i + 1]);
      }
    } else if (ok) {
      float* at = reinterpret_cast<float*>(p.pool) + pool + off;
#pragma unroll
      for (int i = 0; i < N; ++i) at[i * 2 * TD] = u[i];
    }
  }
};

// ---------------------------------------------------------------------------------------------
// Chunk-local state sum  U[i][j] = sum_s w_s v_s[i] conj(k_s[j])  in transposed form, from the key tile AS THE TMA
// DELIVERS IT (interleaved re, im: no operand is built from it) and the value tile split into two weighted planes:
//   A  (MN-major, M = 128 interleaved key columns n' = 2j + c, K = 128 tokens): k'[s][n']   (kr_j at 2j, ki_j at 2j+1)
//   Br (MN-major, N = 64 value channels, K = 128): w_s Re v_s          D1[n'][i] = sum_s A[s][n'] Br[s][i]
//   Bi (                  the same                ): w_s Im v_s          D2[n'][i] = sum_s A[s][n'] Bi[s][i]
//   Re U[i][j] = D1[2j][i] + D2[2j+1][i],   Im U[i][j] = D2[2j][i] - D1[2j+1][i]:  neighbouring TMEM lanes, one shuffle.
// grid = (chunks, H, K); 256 threads; 66 KB shared memory, 128 TMEM columns: three CTAs per SM.
// ---------------------------------------------------------------------------------------------
constexpr size_t OUTER_SMEM = 1024 + 32768 + 32768 + 1536;

// DSTATE == true computes the gradient counterpart  G = sum_t scale e^{A_t} dy_t (x) conj(q_t)  (dy in
// place of v, q in place of k) into dstate slot c.
// The two token tiles (k and v, or q and dy; maps of [B*H*T rows][128 bf16], boxes of 64 x 128, 128-byte swizzle)
// arrive by TMA; the value tile lands in the region its planes are then built in: every thread reads its pieces, a
// barrier, and the planes are written over them.
// FINISH: as p.finish says; the sequences start from zero.
template <bool DSTATE, bool FINISH = false>
__global__ void __launch_bounds__(256, 3) k_tc_chunk_outer(const __grid_constant__ CUtensorMap mk,
                                                           const __grid_constant__ CUtensorMap mv, ScanParams p) {
  using namespace umma;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* sA = smem;            // key tile: [2 boxes of 64 columns][128 rows][128 B]
  unsigned char* sB = smem + 32768;    // value tile, then [256 rows][128 B]: rows s = w Re v_s, rows 128 + s = w Im v_s
  float* Acum = reinterpret_cast<float*>(smem + 65536);          // [128]
  float* wrow = Acum + TC;                                      // [128] weights of the tokens (each is read by 16 threads)
  uint64_t* bar = reinterpret_cast<uint64_t*>(wrow + TC);       // [0] MMAs  [1] token tiles
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + 2);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  pdl_wait();
  const ChunkLoc L = locate_chunk(p.geom, blockIdx.x);
  if (!L.valid) return;
  const int h = blockIdx.y;
  const int kst = blockIdx.z;                 // state (its decay weights the rows); grid z = K
  float graw[4] = {1.f, 1.f, 1.f, 1.f};
  if (warp == 1) warp_cumsum128_load(graw, p.gamma + gamma_base(p, kst, L.b, h, L.t0), L.len, lane);
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    fence_barrier_init();
    const int row0 = (L.b * p.H + h) * p.T + L.t0;
    mbar_arrive_expect_tx(&bar[1], 4 * 16384);
#pragma unroll
    for (int kb = 0; kb < 2; ++kb) {
      tma_load_2d(sA + kb * 16384, &mk, &bar[1], kb * 64, row0);
      tma_load_2d(sB + kb * 16384, &mv, &bar[1], kb * 64, row0);
    }
  }
  __syncwarp();
  if (warp == 0) tmem_alloc<128>(tmem_slot);
  if (warp == 1) warp_cumsum128_finish(Acum, graw, L.len, p.eps, lane);
  tc_fence_before();
  __syncthreads();
  pdl_trigger();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const float a_last = Acum[TC - 1];
  if (tid < TC) wrow[tid] = DSTATE ? p.q_scale * __expf(Acum[tid]) : __expf(fminf(0.f, a_last - Acum[tid]));      // (read behind the next barrier)
  const bool tiles_ok = mbar_wait(&bar[1], 0, 202);
  // this thread's 16-byte pieces of the value tile (rows past the chunk's end belong to someone else: their zeros
  // also cancel whatever the key tile holds in those rows)
  // (rows 16 apart: 2 KB apart in the tile, with the same swizzle)
  const int row0_ = tid >> 4, c16 = tid & 15;
  const unsigned char* src = sB + (c16 >> 3) * 16384 + sw128(row0_, c16 & 7);
  uint4 vxa[8];
#pragma unroll
  for (int it = 0; it < 8; ++it) {
    vxa[it] = make_uint4(0, 0, 0, 0);
    if (row0_ + 16 * it < L.len) vxa[it] = *reinterpret_cast<const uint4*>(src + 2048 * it);
  }
  __syncthreads();      // every piece has been read: the planes may overwrite the tile
  unsigned char* dst_planes = sB + sw128(row0_, c16 >> 1) + (c16 & 1) * 8;
#pragma unroll
  for (int it = 0; it < 8; ++it) {
    const float w = wrow[row0_ + 16 * it];
    const uint32_t vw[4] = {vxa[it].x, vxa[it].y, vxa[it].z, vxa[it].w};
    float vr[4], vi[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 vv = unpack_bf162(vw[e]);
      vr[e] = w * vv.x;
      vi[e] = w * vv.y;
    }
    *reinterpret_cast<uint2*>(dst_planes + 2048 * it) = make_uint2(pack_bf162(vr[0], vr[1]), pack_bf162(vr[2], vr[3]));
    *reinterpret_cast<uint2*>(dst_planes + 16384 + 2048 * it) = make_uint2(pack_bf162(vi[0], vi[1]), pack_bf162(vi[2], vi[3]));
  }
  fence_proxy_async();
  __syncthreads();
  if (warp == 0 && elect_one()) {
    tc_fence_after();
    constexpr uint32_t idesc = idesc_bf16(128, 64, true, true);
    const uint32_t a0 = smem_u32(sA), b0 = smem_u32(sB);
    mma_run(tmem, smem_desc_sw128(a0, 16384, 1024), smem_desc_sw128(b0, 16, 1024), 128, 128, idesc, 8, false);      // D1 = A^T Br: k-step = 16 tokens = 2048 bytes in either operand
    mma_run(tmem + 64, smem_desc_sw128(a0, 16384, 1024), smem_desc_sw128(b0 + 16384, 16, 1024), 128, 128, idesc, 8, false);      // D2 = A^T Bi
    mma_commit(&bar[0]);
  }
  __syncwarp();
  bool ok = mbar_wait(&bar[0], 0, 201) && tiles_ok;
  tc_fence_after();
  {
    // lane n' = 2j+c of the tile holds column i: state[i][j][c] sits at float offset i*128 + n'
    float2* slot = DSTATE ? p.dstates + state_base(p, kst, h, L.slot0 + L.c, TD)
                          : p.states + state_base(p, kst, h, L.slot0 + L.c + 1, TD);
    const int q4 = warp & 3, cc = warp >> 2;   // TMEM lane quarter, column half
    float* dst = reinterpret_cast<float*>(slot) + (q4 * 32 + lane);
    float d1[32], d2[32];
    tmem_ld32(tmem + ((uint32_t)(q4 * 32) << 16) + cc * 32, d1);
    tmem_ld32(tmem + ((uint32_t)(q4 * 32) << 16) + 64 + cc * 32, d2);
    const bool even = (lane & 1) == 0;
    if (FINISH && L.nc == 1) {                  // CTA-uniform
      FinalDest fin;
      fin.init(p, L.seq, pool_slot_of(p, L.seq), kst, h);
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const float o = __shfl_xor_sync(0xffffffffu, d2[i], 1);
        d1[i] = even ? d1[i] + o : o - d1[i];
        if (ok && p.finish == FIN_ALSO) dst[(size_t)(cc * 32 + i) * 128] = d1[i];
      }
      fin.store(p, cc * 32 * 128 + q4 * 32 + lane, d1, even, ok);
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const float other = __shfl_xor_sync(0xffffffffu, d2[i], 1);      // D2 of the neighbouring key column
        const float u = even ? d1[i] + other : other - d1[i];
        if (ok) dst[(size_t)(cc * 32 + i) * 128] = u;
      }
    }
    if (ok && !DSTATE && tid == 0) p.chunk_decay[((size_t)kst * p.H + h) * p.nslots + L.slot0 + L.c + 1] = __expf(a_last);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc<128>(tmem);
  }
}

// ---------------------------------------------------------------------------------------------
// State sums of K states from ONE load of the key / value tiles (2 <= K <= 4).  As in k_tc_chunk_outer
// the key tile is the A operand as the TMA delivers it and the decay weights sit on the value planes, so a state costs
// one rewrite of the planes B_k = w^k_s (Re v_s ; Im v_s) from the registers that hold the value tile, its two MMA
// chains into the same 128 TMEM columns, and its epilogue; the states follow one another.
// grid = (chunks, H); 256 threads; 70 KB shared memory, 128 TMEM columns: three CTAs per SM.
// ---------------------------------------------------------------------------------------------
// DSTATE: the gradient counterpart, G_k = sum_t scale conj(c_kt) e^{A^k_t} dy_t (x) conj(q_t), into dstate slot c.
constexpr size_t OUTERK_SMEM = 1024 + 65536 + KMAX * TC * 12 + 256;

template <bool DSTATE>
__global__ void __launch_bounds__(256, 3) k_tc_chunk_outerK(const __grid_constant__ CUtensorMap mk,
                                                            const __grid_constant__ CUtensorMap mv, ScanParams p) {
  using namespace umma;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* sA = smem;            // key tile: [2 boxes of 64 columns][128 rows][128 B]
  unsigned char* sB = smem + 32768;    // value tile, then per state [256 rows][128 B]: w Re v_s ; w Im v_s
  float* Acum = reinterpret_cast<float*>(smem + 65536);           // [KMAX][128]
  float2* wrow = reinterpret_cast<float2*>(Acum + KMAX * TC);     // DSTATE: [KMAX][128] weight of a token
  uint64_t* bar = reinterpret_cast<uint64_t*>(wrow + KMAX * TC);  // one per state, [KMAX]: the token tiles
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + KMAX + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  pdl_wait();
  const ChunkLoc L = locate_chunk(p.geom, blockIdx.x);
  if (!L.valid) return;
  const int h = blockIdx.y;
  const int K = p.K;
  float graw[4] = {1.f, 1.f, 1.f, 1.f};
  if (warp >= 1 && warp <= K) warp_cumsum128_load(graw, p.gamma + gamma_base(p, warp - 1, L.b, h, L.t0), L.len, lane);
  if (tid == 0) {
    for (int k = 0; k < K; ++k) mbar_init(&bar[k], 1);
    mbar_init(&bar[KMAX], 1);
    fence_barrier_init();
    const int row0 = (L.b * p.H + h) * p.T + L.t0;
    const bool tok = DSTATE && p.dy_tokens;
    mbar_arrive_expect_tx(&bar[KMAX], 4 * 16384);
#pragma unroll
    for (int kb = 0; kb < 2; ++kb) {
      tma_load_2d(sA + kb * 16384, &mk, &bar[KMAX], kb * 64, row0);
      tma_load_2d(sB + kb * 16384, &mv, &bar[KMAX], (tok ? h * 128 : 0) + kb * 64, tok ? L.b * p.T + L.t0 : row0);
    }
  }
  __syncwarp();
  if (warp == 0) tmem_alloc<128>(tmem_slot);
  if (warp >= 1 && warp <= K) warp_cumsum128_finish(Acum + (warp - 1) * TC, graw, L.len, p.eps, lane);
  tc_fence_before();
  __syncthreads();
  pdl_trigger();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  for (int e = tid; e < K * TC; e += 256) {          // (read after the barrier in front of the first planes)
    const int k = e / TC, t = e - k * TC;
    if (!DSTATE) {
      wrow[e].x = __expf(fminf(0.f, Acum[k * TC + TC - 1] - Acum[e]));
    } else {
      float2 c = make_float2(1.f, 0.f);
      if (p.coef != nullptr && t < L.len) c = __ldg(reinterpret_cast<const float2*>(p.coef + gamma_base(p, k, L.b, h, L.t0 + t) * 2));
      const float f = p.q_scale * __expf(Acum[e]);
      wrow[e] = make_float2(c.x * f, -c.y * f);
    }
  }
  bool ok = mbar_wait(&bar[KMAX], 0, 206);
  // this thread's 16-byte pieces of the value tile (rows past the chunk's end: zeros, which also cancel whatever the
  // key tile holds in those rows)
  // (rows 16 apart: 2 KB apart in the tile, with the same swizzle)
  const int row0_ = tid >> 4, c16 = tid & 15;
  const unsigned char* src = sB + (c16 >> 3) * 16384 + sw128(row0_, c16 & 7);
  unsigned char* dst_planes = sB + sw128(row0_, c16 >> 1) + (c16 & 1) * 8;
  uint4 vxa[8];
#pragma unroll
  for (int it = 0; it < 8; ++it) {
    vxa[it] = make_uint4(0, 0, 0, 0);
    if (row0_ + 16 * it < L.len) vxa[it] = *reinterpret_cast<const uint4*>(src + 2048 * it);
  }
  const int q4 = warp & 3, cc = warp >> 2;   // epilogue: TMEM lane quarter, column half
  const bool even = (lane & 1) == 0;
  __syncthreads();      // every piece has been read
  // A state's planes are written as soon as the previous one's MMAs have read theirs, and the previous one's sums leave the accumulators
  // after that: one barrier a state, and the passes of different warps overlap.  With the sums in groups of 8 columns (the value tile
  // stays in registers beside them) 48 chat prompts took 310 instead of 322 us, 8 x 6 x 2048 with three states 395 instead of 398.
#pragma unroll 1
  for (int k = 0; k <= K; ++k) {
    if (k < K) {
#pragma unroll
      for (int it = 0; it < 8; ++it) {
        const uint4 vx = vxa[it];
        const float2 w = DSTATE ? wrow[k * TC + row0_ + 16 * it] : make_float2(wrow[k * TC + row0_ + 16 * it].x, 0.f);
        const uint32_t vw[4] = {vx.x, vx.y, vx.z, vx.w};
        float vr[4], vi[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 vv = unpack_bf162(vw[e]);
          vr[e] = DSTATE ? w.x * vv.x - w.y * vv.y : w.x * vv.x;
          vi[e] = DSTATE ? w.x * vv.y + w.y * vv.x : w.x * vv.y;
        }
        *reinterpret_cast<uint2*>(dst_planes + 2048 * it) = make_uint2(pack_bf162(vr[0], vr[1]), pack_bf162(vr[2], vr[3]));
        *reinterpret_cast<uint2*>(dst_planes + 16384 + 2048 * it) = make_uint2(pack_bf162(vi[0], vi[1]), pack_bf162(vi[2], vi[3]));
      }
    }
    if (k > 0) {
      // Re U = D1[2j] + D2[2j+1], Im U = D2[2j] - D1[2j+1]: lane n' = 2j+c holds column i, state[i][j][c] at i*128 + n'
      float2* slot = DSTATE ? p.dstates + state_base(p, k - 1, h, L.slot0 + L.c, TD) : p.states + state_base(p, k - 1, h, L.slot0 + L.c + 1, TD);
      float* dst = reinterpret_cast<float*>(slot) + (q4 * 32 + lane);
      const bool final_now = !DSTATE && p.finish != FIN_NONE && L.nc == 1;
#pragma unroll 1
      for (int hh = 0; hh < 4; ++hh) {          // 8 columns at a time
        float d1[8], d2[8];
        const uint32_t col = (uint32_t)(cc * 32 + hh * 8);
        tmem_ld8x2(tmem + ((uint32_t)(q4 * 32) << 16) + col, d1, tmem + ((uint32_t)(q4 * 32) << 16) + 64 + col, d2);
        if (final_now) {
          FinalDest fin;
          fin.init(p, L.seq, pool_slot_of(p, L.seq), k - 1, h);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float o = __shfl_xor_sync(0xffffffffu, d2[i], 1);
            d1[i] = even ? d1[i] + o : o - d1[i];
            if (ok && p.finish == FIN_ALSO) dst[(size_t)(col + i) * 128] = d1[i];
          }
          fin.store(p, (int)col * 128 + q4 * 32 + lane, d1, even, ok);
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float other = __shfl_xor_sync(0xffffffffu, d2[i], 1);
            const float u = even ? d1[i] + other : other - d1[i];
            if (ok) dst[(size_t)(col + i) * 128] = u;
          }
        }
      }
      if (ok && !DSTATE && tid == 0) p.chunk_decay[((size_t)(k - 1) * p.H + h) * p.nslots + L.slot0 + L.c + 1] = __expf(Acum[(k - 1) * TC + TC - 1]);
    }
    if (k == K) break;
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    if (warp == 0 && elect_one()) {
      tc_fence_after();
      constexpr uint32_t idesc = idesc_bf16(128, 64, true, true);
      const uint32_t a0 = smem_u32(sA), b0 = smem_u32(sB);
      mma_run(tmem, smem_desc_sw128(a0, 16384, 1024), smem_desc_sw128(b0, 16, 1024), 128, 128, idesc, 8, false);      // D1 = A^T Br
      mma_run(tmem + 64, smem_desc_sw128(a0, 16384, 1024), smem_desc_sw128(b0 + 16384, 16, 1024), 128, 128, idesc, 8, false);      // D2 = A^T Bi
      mma_commit(&bar[k]);
    }
    __syncwarp();
    ok = mbar_wait(&bar[k], 0, 205) && ok;
    tc_fence_after();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc<128>(tmem);
  }
}

enum ChunkMode { M_FWD = 0, M_DQ = 1, M_DV = 2, M_DK = 3, M_ANY = 4 };

struct ChunkMaps {
  CUtensorMap a1, b1, x2;  // [B*H*T rows][128 bf16], boxes of 64 x 128, 128-byte swizzle
  CUtensorMap out;         // the output tensor, same shape, boxes of 64 x 32 (one per epilogue warp)
};

}  // namespace tcs
}  // namespace qpam
