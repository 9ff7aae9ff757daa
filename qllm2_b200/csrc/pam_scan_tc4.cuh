// Backward of the chunked PAM scan on tensor cores for 2 <= K <= 4 phase-routed states: ALL gradients of a 128-token chunk,
// for every state, in one CTA (bf16 token tensors, head dim 64).  With A^k the cumulative log decay of state k inside the chunk,
// D^k_ts = e^{A^k_t - A^k_s} (s <= t < len), c_k the read-out weights, sigma the query scale:
//
//   X_ts = dy_t . conj(v_s)      Y_ts = q_t . conj(k_s)      G_ts = sigma sum_k conj(c_kt) D^k_ts
//   dq_t = sum_s (G X)_ts k_s                 + sum_k sigma conj(c_kt) e^{A^k_t} (S^k_c)^H dy_t
//   dk_s = sum_t conj((G X)_ts) q_t           + sum_k e^{A^k_last - A^k_s} (dS^k_c+1)^H v_s
//   dv_s = sum_t (G conj(Y))_ts dy_t          + sum_k e^{A^k_last - A^k_s} dS^k_c+1 k_s
//   dc_kt        = sigma [ sum_s D^k_ts Z_ts + e^{A^k_t} conj(q_t) . (S^k_c)^H dy_t ],     Z_ts = X_ts conj(Y_ts)
//   Re<q,dq>_kt  = Re(conj(c_kt) dc_kt)
//   Re<k,dk>_ks  = sigma sum_t D^k_ts Re(conj(c_kt) Z_ts) + e^{A^k_last - A^k_s} Re<k_s, (dS^k_c+1)^H v_s>
//
// The scores do not depend on the state, so K states cost one pass of the tile products; what a state adds is its term of
// the weight G, its sums of Z and its carried-state products.  dc and the decay gradient come from the fp32 scores (no
// per-state output is needed, and the contribution of every (t, s) pair to Re<q,dq> - Re<k,dk> cancels to fp32 rounding).
// (One state keeps the three-job kernel of pam_scan_tc2.cuh: two CTAs on an SM hide each other's waits there, 102-106 us against
// 118 us here at 8 x 6 x 2048 (93 now); three states took 420 us that way, read-out weights included, and take 214 us.)
//
// Every score is formed twice, once per direction of the sum (a row of the tile is a TMEM lane, so sums along a row stay
// inside threads): pass A has tokens t as rows (dq, dc), pass B tokens s (dk, dv, Re<k,dk>).  512 threads: a thread owns a
// row and 32 columns of both score tiles in a pass and 16 channels of its row in the outputs.
//
//   TMEM        [0,128)              [128,256)           [256,384)            [384,512)
//   scores      X real               X imaginary         Y real               Y imaginary
//   dq          G X (bf16)           dq accumulator      (S^0)^H dy           (S^1)^H dy     (then state 2 in [0,128), 3 in [256,384))
//   scores      X^H real             X^H imaginary       Y^H real             Y^H imaginary
//   dk, dv      conj(G X)^T (bf16)   dk accumulator      (G conj Y)^T (bf16)  dv accumulator
//   carried     (dS^0)^H v           (dS^1)^H v          dS^0 k               dS^1 k         (then states 2, 3)
//
// Decay: D factors as e^{A_t - A_m} e^{A_m - A_s} around the middle of the chunk; a state whose chunk decays by more than
// e^-80 takes one exponential per score instead (see pam_scan_tc2.cuh).
#pragma once
#include "pam_scan_tc2.cuh"

namespace qpam {
namespace tcs {

constexpr int BT = 512;                    // threads
constexpr size_t BWDK_SMEM = 1024 + 4 * 32768 + 4 * 16384 + KMAX * TC * (4 + 4 + 8 + 4) + 4 * KMAX * TC * 8 + 256;

// acc (real parts at acc, imaginary at acc + 64) = A (.) state planes, as bw_issue_state
template <bool OP_H>
__device__ __forceinline__ void issue_state(uint32_t acc, uint32_t a_r, uint32_t s_r) { bw_issue_state(OP_H, acc - 128, a_r, s_r, false); }

// acc = T X2, T's packed scores in the columns its fp32 scores had: of every 16 columns the first 8 hold the real parts
__device__ __forceinline__ void issue_rows(uint32_t t, uint32_t acc, uint32_t x_r) {
  using namespace umma;
  constexpr uint32_t id = idesc_bf16(128, 64, false, true);
  constexpr uint32_t idn = idesc_bf16_nega(128, 64, false, true);
  constexpr uint32_t id2 = idesc_bf16(128, 128, false, true);      // (both planes of X2 as one B operand: N blocks 16 KB apart)
  mma_run_ts(acc, t, smem_desc_sw128(x_r, 16384, 1024), 16, 128, id2, 8, false);
  mma_run_ts(acc, t + 8, smem_desc_sw128(x_r + 16384, 16, 1024), 16, 128, idn, 8, true);
  mma_run_ts(acc + 64, t + 8, smem_desc_sw128(x_r, 16, 1024), 16, 128, id, 8, true);
}

struct BwdTables {
  float* A;        // [K][128] cumulative log decay
  float* col;      // [K][128] e^{A_m - A_s}                       (strong: 1)
  float* row;      // [K][128] sigma e^{A_t - A_m}, 0 past the end (strong: sigma)
  float *wr, *wi;  // [K][128] conj(c_t) row_t
};

// Pass A for 16 columns of row r: T = G X over the columns of X, sums of col_s D Z over the columns into zs (real and imaginary, even
// and odd columns apart).
template <int K, bool STRONG>
__device__ __forceinline__ void pass_a16(uint32_t tl, int c0, int q4, int r, const BwdTables& tb, uint32_t strong, const float2 (&wk)[K],
                                         float2 (&zs)[K][2]) {
  using namespace umma;
  uint32_t out[16];
  if (c0 > q4 * 32 + 31) {                  // warp-uniform: above the diagonal
#pragma unroll
    for (int j = 0; j < 16; ++j) out[j] = 0u;
  } else {
    uint32_t xr[16], xi[16], yr[16], yi[16];
    tmem_ld16x4(tl + c0, xr, tl + 128 + c0, xi, tl + 256 + c0, yr, tl + 384 + c0, yi);
    const int last = c0 + 15 <= q4 * 32 ? TC : r;      // no diagonal inside the block: every column counts
#pragma unroll
    for (int j = 0; j < 16; j += 2) {          // two columns an instruction
      const int c1 = c0 + j;
      const float2 x = make_float2(__uint_as_float(xr[j]), __uint_as_float(xr[j + 1])), y = make_float2(__uint_as_float(xi[j]), __uint_as_float(xi[j + 1]));
      const float2 u = make_float2(__uint_as_float(yr[j]), __uint_as_float(yr[j + 1])), v = make_float2(__uint_as_float(yi[j]), __uint_as_float(yi[j + 1]));
      float2 cf[K], gr = make_float2(0.f, 0.f), gi = gr;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        cf[k] = *reinterpret_cast<const float2*>(tb.col + k * TC + c1);
        if (STRONG && ((strong >> k) & 1u)) cf[k] = make_float2(__expf(fminf(0.f, tb.A[k * TC + r] - tb.A[k * TC + c1])), __expf(fminf(0.f, tb.A[k * TC + r] - tb.A[k * TC + c1 + 1])));
        gr = ffma2(make_float2(wk[k].x, wk[k].x), cf[k], gr);
        gi = ffma2(make_float2(wk[k].y, wk[k].y), cf[k], gi);
      }
      const float2 xv = fmul2(x, v);
      float2 zr = ffma2(x, u, fmul2(y, v)), zi = ffma2(y, u, make_float2(-xv.x, -xv.y));
      if (c1 > last) gr.x = gi.x = zr.x = zi.x = 0.f;
      if (c1 + 1 > last) gr.y = gi.y = zr.y = zi.y = 0.f;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        zs[k][0] = ffma2(cf[k], zr, zs[k][0]);
        zs[k][1] = ffma2(cf[k], zi, zs[k][1]);
      }
      const float2 iy = fmul2(gi, y);
      const float2 tr = ffma2(gr, x, make_float2(-iy.x, -iy.y)), ti = ffma2(gr, y, fmul2(gi, x));
      out[j >> 1] = pack_bf162(tr.x, tr.y);
      out[8 + (j >> 1)] = pack_bf162(ti.x, ti.y);
    }
  }
  tmem_st16(tl + c0, out);
}

// Pass B for 16 columns (tokens t) of row s = r: conj(G X)^T over the columns of X^H, (G conj Y)^T over those of Y^H, sums
// of sigma e^{A_t - A_m} Re(conj(c) Z) into cs.
template <int K, bool STRONG>
__device__ __forceinline__ void pass_b16(uint32_t tl, int c0, int q4, int r, const BwdTables& tb, uint32_t strong, const float (&ck)[K],
                                         float2 (&cs)[K]) {
  using namespace umma;
  uint32_t ox[16], oy[16];
  if (c0 + 15 < q4 * 32) {
#pragma unroll
    for (int j = 0; j < 16; ++j) ox[j] = oy[j] = 0u;
  } else {
    uint32_t xr[16], xi[16], yr[16], yi[16];
    tmem_ld16x4(tl + c0, xr, tl + 128 + c0, xi, tl + 256 + c0, yr, tl + 384 + c0, yi);
    const int first = c0 >= q4 * 32 + 31 ? 0 : r;
#pragma unroll
    for (int j = 0; j < 16; j += 2) {          // two columns an instruction
      const int c1 = c0 + j;
      const float2 x = make_float2(__uint_as_float(xr[j]), __uint_as_float(xr[j + 1])), y = make_float2(__uint_as_float(xi[j]), __uint_as_float(xi[j + 1]));
      const float2 u = make_float2(__uint_as_float(yr[j]), __uint_as_float(yr[j + 1])), v = make_float2(__uint_as_float(yi[j]), __uint_as_float(yi[j + 1]));
      float2 wr[K], wi[K], gr = make_float2(0.f, 0.f), gi = gr;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        wr[k] = *reinterpret_cast<const float2*>(tb.wr + k * TC + c1);
        wi[k] = *reinterpret_cast<const float2*>(tb.wi + k * TC + c1);
        if (STRONG && ((strong >> k) & 1u)) {
          const float2 f = make_float2(__expf(fminf(0.f, tb.A[k * TC + c1] - tb.A[k * TC + r])), __expf(fminf(0.f, tb.A[k * TC + c1 + 1] - tb.A[k * TC + r])));
          wr[k] = fmul2(wr[k], f);
          wi[k] = fmul2(wi[k], f);
        }
        gr = ffma2(wr[k], make_float2(ck[k], ck[k]), gr);
        gi = ffma2(wi[k], make_float2(ck[k], ck[k]), gi);
      }
      const float2 xv = fmul2(x, v);
      float2 zr = ffma2(x, u, fmul2(y, v)), zn = ffma2(y, u, make_float2(-xv.x, -xv.y));      // conj(X^H) Y^H: the real part, the imaginary part negated
      if (c1 < first) gr.x = gi.x = zr.x = zn.x = 0.f;
      if (c1 + 1 < first) gr.y = gi.y = zr.y = zn.y = 0.f;
#pragma unroll
      for (int k = 0; k < K; ++k) cs[k] = ffma2(wr[k], zr, ffma2(wi[k], zn, cs[k]));
      const float2 ix = fmul2(gi, x), iv = fmul2(gi, v);
      const float2 xo = ffma2(gr, x, fmul2(gi, y)), xp = ffma2(gr, y, make_float2(-ix.x, -ix.y));
      const float2 yo = ffma2(gr, u, make_float2(-iv.x, -iv.y)), yp = ffma2(gr, v, fmul2(gi, u));
      ox[j >> 1] = pack_bf162(xo.x, xo.y);
      ox[8 + (j >> 1)] = pack_bf162(xp.x, xp.y);
      oy[j >> 1] = pack_bf162(yo.x, yo.y);
      oy[8 + (j >> 1)] = pack_bf162(yp.x, yp.y);
    }
  }
  tmem_st16(tl + c0, ox);
  tmem_st16(tl + 256 + c0, oy);
}

// carried state (fp32 [64][64] re, im) -> bf16 planes of a slot; a warp's 512 consecutive bytes are one row
__device__ __forceinline__ void state_load(float4 (&v)[4], const float2* state, int tid) {
  const float4* sg = reinterpret_cast<const float4*>(state);
#pragma unroll
  for (int it = 0; it < 4; ++it) v[it] = ld_dependent(sg + tid + BT * it);
}
__device__ __forceinline__ void state_stage(unsigned char* slot, const float4 (&v)[4], int tid) {
#pragma unroll
  for (int it = 0; it < 4; ++it) {
    const int i = (tid + BT * it) >> 5, c = tid & 31;      // row i, columns 2c and 2c + 1
    const uint32_t off = sw128(i, c >> 2) + (c & 3) * 4;
    *reinterpret_cast<uint32_t*>(slot + off) = pack_bf162(v[it].x, v[it].z);
    *reinterpret_cast<uint32_t*>(slot + 8192 + off) = pack_bf162(v[it].y, v[it].w);
  }
}

// 16 channels of row r (channels [16 cq, 16 cq + 16)) of a de-interleaved tile
__device__ __forceinline__ void row16(const unsigned char* planes, int r, int cq, float (&re)[16], float (&im)[16]) {
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    const uint4 a = *reinterpret_cast<const uint4*>(planes + sw128(r, 2 * cq + g)), b = *reinterpret_cast<const uint4*>(planes + 16384 + sw128(r, 2 * cq + g));
    const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 x = unpack_bf162(aw[e]), y = unpack_bf162(bw[e]);
      re[g * 8 + 2 * e] = x.x; re[g * 8 + 2 * e + 1] = x.y;
      im[g * 8 + 2 * e] = y.x; im[g * 8 + 2 * e + 1] = y.y;
    }
  }
}

// 16 finished channels of a row: into the staging block [2 boxes of 32 channels][128 rows][128 B] of a TMA store, or (a
// ragged chunk: rows past the end belong to someone else) straight to global memory
__device__ __forceinline__ void put16(const float (&re)[16], const float (&im)[16], unsigned char* stage, __nv_bfloat16* __restrict__ row, int r, int cq,
                                      bool bulk, bool valid) {
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    const uint4 pk = make_uint4(pack_bf162(re[4 * g], im[4 * g]), pack_bf162(re[4 * g + 1], im[4 * g + 1]), pack_bf162(re[4 * g + 2], im[4 * g + 2]),
                          pack_bf162(re[4 * g + 3], im[4 * g + 3]));
    if (bulk) {
      *reinterpret_cast<uint4*>(stage + (cq >> 1) * 16384 + r * 128 + (((4 * (cq & 1) + g) ^ (r & 7)) << 4)) = pk;
    } else if (valid) {
      *reinterpret_cast<uint4*>(row + cq * 32 + g * 8) = pk;
    }
  }
}
// box b (0..7: 32 rows of 32 channels) of a staging block leaves by TMA; one thread
__device__ __forceinline__ void store_box(const CUtensorMap* map, const unsigned char* stage, int b, int row0) {
  const unsigned char* box = stage + (b >> 2) * 16384 + (b & 3) * 4096;
  umma::tma_store_2d_keep(map, box, (b >> 2) * 64, row0 + (b & 3) * 32);
}

// grid = (chunks, H)
template <int K>
__global__ void __launch_bounds__(BT, 1) k_tc_scan_bwdK(const __grid_constant__ BwdMaps maps, ScanParams p, const float* __restrict__ anchor_parts) {
  using namespace umma;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char *TQ = smem, *TK = TQ + 32768, *TV = TK + 32768, *TY = TV + 32768;      // q, k, v, dy: real plane, imaginary plane
  unsigned char* SL = TY + 32768;                                                     // 4 slots of carried-state planes, 16 KB each
  BwdTables tb;
  tb.A = reinterpret_cast<float*>(SL + 4 * 16384);
  tb.col = tb.A + KMAX * TC;
  tb.wr = tb.col + KMAX * TC;
  tb.wi = tb.wr + KMAX * TC;
  tb.row = tb.wi + KMAX * TC;
  float2* dcp = reinterpret_cast<float2*>(tb.row + KMAX * TC);      // [4 channel groups][K][128] shares of dc
  float* kdp = reinterpret_cast<float*>(SL + 2 * 16384);            // [4][K][128] shares of Re<k, dk>, once no MMA reads the slots
  uint64_t* bars = reinterpret_cast<uint64_t*>(dcp + 4 * KMAX * TC);
  enum { B_VY, B_QK, B_SA, B_SB, B_DQ, B_U2, B_U3, B_DKV, B_C0, B_C1, B_C2, B_C3, N_BARS };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + N_BARS);
  int* failed = reinterpret_cast<int*>(tmem_slot + 1);
  float* wsum = reinterpret_cast<float*>(failed + 1);               // [K][4]
  float* anc = wsum + 4 * KMAX;                                     // [K][2]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const ChunkLoc L = locate_chunk(p.geom, blockIdx.x);
  if (!L.valid) {
    pdl_wait();
    return;
  }
  const int h = blockIdx.y, len = L.len;
  const bool has_s = L.c > 0 || p.s0 != nullptr, has_ds = L.c < L.nc - 1 || p.ds_final != nullptr;
  const int row0 = (L.b * p.H + h) * p.T + L.t0;
  if (tid == BT - 1) *failed = device_error_now();
  float graw[4] = {1.f, 1.f, 1.f, 1.f};
  if (warp >= 1 && warp <= K) warp_cumsum128_load(graw, p.gamma + gamma_base(p, warp - 1, L.b, h, L.t0), len, lane);
  if (tid == 0) {
#pragma unroll
    for (int i = 0; i < N_BARS; ++i) mbar_init(&bars[i], 1);
    fence_barrier_init();
    const int dx = p.dy_tokens ? h * 128 : 0, dr = p.dy_tokens ? L.b * p.T + L.t0 : row0;
    mbar_arrive_expect_tx(&bars[B_VY], 4 * 16384);
#pragma unroll
    for (int kb = 0; kb < 2; ++kb) {
      tma_load_2d(TY + kb * 16384, &maps.dy, &bars[B_VY], dx + kb * 64, dr);
      tma_load_2d(TV + kb * 16384, &maps.v, &bars[B_VY], kb * 64, row0);
    }
    if (has_s) {
#pragma unroll
      for (int k = 0; k < K; ++k) bulk_prefetch_l2(p.states + state_base(p, k, h, L.slot0 + L.c, TD), 32768);
    }
    mbar_arrive_expect_tx(&bars[B_QK], 4 * 16384);
#pragma unroll
    for (int kb = 0; kb < 2; ++kb) {
      tma_load_2d(TQ + kb * 16384, &maps.q, &bars[B_QK], kb * 64, row0);
      tma_load_2d(TK + kb * 16384, &maps.k, &bars[B_QK], kb * 64, row0);
    }
  }
  __syncwarp();
  const int ek = tid >> 7, et = tid & 127;          // this thread's (state, token) in the tables
  const size_t eg = gamma_base(p, ek, L.b, h, L.t0 + et);
  float2 c_e = make_float2(1.f, 0.f);
  if (p.coef != nullptr && ek < K && et < len) c_e = __ldg(reinterpret_cast<const float2*>(p.coef + eg * 2));
  // what the decay gradient needs at the end, requested as soon as it may be: the decay of this thread's token, and (further
  // down, they are the predecessor's) per state the partial sums of the anchors at the chunk's first token and just after the
  // chunk (two warps of the state's four)
  const int et_rev = TC - 1 - et;
  float g_e = 1.f, an0 = 0.f, an1 = 0.f;
  if (ek < K && et_rev < len) g_e = __ldg(p.gamma + eg - et + et_rev);
  if (warp == 0) tmem_alloc<512>(tmem_slot);
  if (warp >= 1 && warp <= K) warp_cumsum128_finish(tb.A + (warp - 1) * TC, graw, len, p.eps, lane);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_trigger();
  const uint32_t tmem = *tmem_slot;
  if (*failed != 0) {       // an earlier launch gave up on a wait: outputs stay untouched (the tiles still have to land)
    pdl_wait();
    mbar_wait(&bars[B_VY], 0, 250);
    mbar_wait(&bars[B_QK], 0, 250);
    __syncthreads();
    if (warp == 0) tmem_dealloc<512>(tmem);
    return;
  }
  uint32_t strong = 0;
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (tb.A[k * TC + TC - 1] < STRONG_DECAY) strong |= 1u << k;
  if (ek < K) {
    const bool st = (strong >> ek) & 1u;
    const float a = tb.A[ek * TC + et], a_mid = tb.A[ek * TC + TC / 2 - 1];
    const float rf = et < len ? p.q_scale * (st ? 1.f : __expf(a - a_mid)) : 0.f;
    tb.col[ek * TC + et] = st ? 1.f : __expf(a_mid - a);
    tb.row[ek * TC + et] = rf;
    tb.wr[ek * TC + et] = c_e.x * rf;
    tb.wi[ek * TC + et] = -c_e.y * rf;
  }
  const uint32_t q_r = smem_u32(TQ), k_r = smem_u32(TK), v_r = smem_u32(TV), y_r = smem_u32(TY), sl = smem_u32(SL);
  const bool issuer = warp == 0 && elect_one();
  // the states entering the chunk, while the tiles are on their way
  // the carried states of two states are in flight while the tiles are de-interleaved, the others while those are staged
  float4 sv[2][4];
  auto load_state = [&](int k) { state_load(sv[k & 1], p.states + state_base(p, k, h, L.slot0 + L.c, TD), tid); };
  if (has_s) {
    load_state(0);
    load_state(1);
  }
  // de-interleave dy and v, start X; then q and k, start Y
  bool ok = mbar_wait(&bars[B_VY], 0, 251);
  {
    const int row = tid & 127, hb = (tid >> 7) & 1;
    unsigned char* tile = tid < 256 ? TY : TV;
    uint4 ra[8];
    deint_read(tile, row, hb, ra);
    __syncthreads();
    deint_write(tile, row, hb, ra);
    fence_proxy_async();
    __syncthreads();
    if (issuer) bw_issue_scores(tmem, y_r, v_r);
    __syncwarp();
    if (has_s) {
      state_stage(SL, sv[0], tid);
      if (K > 2) load_state(2);
      state_stage(SL + 16384, sv[1], tid);
      if (K > 3) load_state(3);
    }
    ok = mbar_wait(&bars[B_QK], 0, 252) && ok;
    tile = tid < 256 ? TQ : TK;
    deint_read(tile, row, hb, ra);
    __syncthreads();
    deint_write(tile, row, hb, ra);
    fence_proxy_async();
    __syncthreads();
    if (issuer) {
      bw_issue_scores(tmem + 256, q_r, k_r);
      mma_commit(&bars[B_SA]);
    }
    __syncwarp();
    if (has_s) {
      if (K > 2) state_stage(SL + 2 * 16384, sv[0], tid);
      if (K > 3) state_stage(SL + 3 * 16384, sv[1], tid);
    }
  }
  const int q4 = warp & 3, cq = warp >> 2;
  const int r = q4 * 32 + lane;                                   // this thread's row (TMEM lane)
  const uint32_t tl = tmem + ((uint32_t)(q4 * 32) << 16);
  const bool valid = r < len;
  const size_t obase = token_base(p, L.b, h, L.t0 + r, TD);

  if (tid == 0 && has_ds) {      // (a hint: the reverse carry may still be writing them)
#pragma unroll
    for (int k = 0; k < K; ++k) bulk_prefetch_l2(p.dstates + state_base(p, k, h, L.slot0 + L.c + 1, TD), 32768);
  }
  // ---- pass A: rows t
  float2 wk[K], zp[K][2], zs[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    wk[k] = make_float2(tb.wr[k * TC + r], tb.wi[k * TC + r]);
    zp[k][0] = zp[k][1] = make_float2(0.f, 0.f);
  }
  ok = mbar_wait(&bars[B_SA], 0, 253) && ok;
  tc_fence_after();
#pragma unroll 1
  for (int hh = 0; hh < 2; ++hh) {
    const int c0 = cq * 32 + hh * 16;
    if (strong == 0u) pass_a16<K, false>(tl, c0, q4, r, tb, 0u, wk, zp);
    else pass_a16<K, true>(tl, c0, q4, r, tb, strong, wk, zp);
  }
#pragma unroll
  for (int k = 0; k < K; ++k) zs[k] = make_float2(zp[k][0].x + zp[k][0].y, zp[k][1].x + zp[k][1].y);
  tmem_st_wait();
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  if (issuer) {
    tc_fence_after();
    issue_rows(tmem, tmem + 128, k_r);
    if (has_s) {
      issue_state<true>(tmem + 256, y_r, sl);
      issue_state<true>(tmem + 384, y_r, sl + 16384);
    }
    mma_commit(&bars[B_DQ]);
    if (K > 2 && has_s && mbar_wait(&bars[B_DQ], 0, 254)) {        // the packed scores have been consumed: state 2 takes their columns
      issue_state<true>(tmem, y_r, sl + 2 * 16384);
      mma_commit(&bars[B_U2]);
    }
  }
  __syncwarp();
  ok = mbar_wait(&bars[B_DQ], 0, 254) && ok;
  tc_fence_after();
  {
    float vr[16], vi[16];
    tmem_ld16x2(tl + 128 + 16 * cq, vr, tl + 192 + 16 * cq, vi);
    if (has_s) {
#pragma unroll
      for (int k = 0; k < K; ++k) {
        if (K > 3 && k == 1) {              // state 0's accumulator has been read: state 3 takes it
          tc_fence_before();
          __syncthreads();
          if (issuer) {
            tc_fence_after();
            issue_state<true>(tmem + 256, y_r, sl + 3 * 16384);
            mma_commit(&bars[B_U3]);
          }
          __syncwarp();
        }
        if (k >= 2) {
          ok = mbar_wait(&bars[k == 2 ? B_U2 : B_U3], 0, 255) && ok;
          tc_fence_after();
        }
        const uint32_t at = tl + (k == 2 ? 0 : k == 1 ? 384 : 256) + 16 * cq;
        float ur[16], ui[16], xr[16], xi[16];
        tmem_ld16x2(at, ur, at + 64, ui);
        row16(TQ, r, cq, xr, xi);
        const float f = __expf(((strong >> k) & 1u) ? tb.A[k * TC + r] : tb.A[k * TC + TC / 2 - 1]);      // row_t f = sigma e^{A_t}
        const float wr = wk[k].x * f, wi = wk[k].y * f;
        float2 er = make_float2(0.f, 0.f), ei = er, en = er;      // (two channels an instruction; ei - en is the imaginary part)
        const float2 wr2 = make_float2(wr, wr), wi2 = make_float2(wi, wi), wn2 = make_float2(-wi, -wi);
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          const float2 a = make_float2(ur[j], ur[j + 1]), b = make_float2(ui[j], ui[j + 1]), c = make_float2(xr[j], xr[j + 1]), d = make_float2(xi[j], xi[j + 1]);
          er = ffma2(c, a, ffma2(d, b, er));
          ei = ffma2(c, b, ei);
          en = ffma2(d, a, en);
          const float2 o = ffma2(wr2, a, ffma2(wn2, b, make_float2(vr[j], vr[j + 1]))), p2 = ffma2(wr2, b, ffma2(wi2, a, make_float2(vi[j], vi[j + 1])));
          vr[j] = o.x; vr[j + 1] = o.y;
          vi[j] = p2.x; vi[j + 1] = p2.y;
        }
        zs[k].x = fmaf(f, er.x + er.y, zs[k].x);
        zs[k].y = fmaf(f, (ei.x - en.x) + (ei.y - en.y), zs[k].y);
      }
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const float rw = tb.row[k * TC + r];
      dcp[(cq * K + k) * TC + r] = make_float2(rw * zs[k].x, rw * zs[k].y);
    }
    tc_fence_before();
    __syncthreads();                        // accumulators and state slots have been read
    if (issuer) {
      tc_fence_after();
      bw_issue_scores(tmem, v_r, y_r);
      bw_issue_scores(tmem + 256, k_r, q_r);
      mma_commit(&bars[B_SB]);
    }
    __syncwarp();
    put16(vr, vi, SL, reinterpret_cast<__nv_bfloat16*>(p.dq) + obase, r, cq, len == TC, valid && ok);
  }
  fence_proxy_async();
  __syncthreads();
  const bool storing = warp >= 8 && lane == 0 && len == TC && ok;
  if (storing) store_box(&maps.dq, SL, warp - 8, row0);
  float4 gv[2][4];
  auto load_grad = [&](int k) { state_load(gv[k & 1], p.dstates + state_base(p, k, h, L.slot0 + L.c + 1, TD), tid); };
  auto stage_grad = [&](int k) { state_stage(SL + ((k + 2) & 3) * 16384, gv[k & 1], tid); };
  // the gradients of the states and the anchors are the reverse carry's; everything above is the call's inputs and the forward
  // states, which are older (see launch_after)
  pdl_wait();
  if (ek < K && (warp & 3) < 2 && anchor_parts != nullptr) {      // (null: zero, see scan_bwd_tc)
    const float* ap = anchor_parts + (((size_t)ek * p.H + h) * p.nslots + L.slot0 + L.c + (warp & 3)) * ANCHOR_PARTS;
    an0 = __ldcg(ap + lane);
    an1 = __ldcg(ap + lane + 32);
  }
  if (has_ds) {
    load_grad(0);
    load_grad(1);
    stage_grad(0);
    if (K > 2) load_grad(2);
    stage_grad(1);
    if (K > 3) load_grad(3);
  }
  if (K > 2) {
    if (storing) tma_store_wait_read();
    __syncthreads();                        // the staging block has left: slots 0 and 1 are free
    if (has_ds) {
      stage_grad(2);
      if (K > 3) stage_grad(3);
    }
  }

  // ---- pass B: rows s
  float ck[K], cs[K];
  float2 cp[K];                             // even and odd columns apart
#pragma unroll
  for (int k = 0; k < K; ++k) {
    ck[k] = tb.col[k * TC + r];
    cp[k] = make_float2(0.f, 0.f);
  }
  ok = mbar_wait(&bars[B_SB], 0, 256) && ok;
  tc_fence_after();
#pragma unroll 1
  for (int hh = 0; hh < 2; ++hh) {
    const int c0 = cq * 32 + hh * 16;
    if (strong == 0u) pass_b16<K, false>(tl, c0, q4, r, tb, 0u, ck, cp);
    else pass_b16<K, true>(tl, c0, q4, r, tb, strong, ck, cp);
  }
  tmem_st_wait();
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  if (issuer) {
    tc_fence_after();
    issue_rows(tmem, tmem + 128, q_r);
    issue_rows(tmem + 256, tmem + 384, y_r);
    mma_commit(&bars[B_DKV]);
    if (has_ds && mbar_wait(&bars[B_DKV], 0, 257)) {       // the packed scores have been consumed: state 0 takes their columns
      issue_state<true>(tmem, v_r, sl + 2 * 16384);
      issue_state<false>(tmem + 256, k_r, sl + 2 * 16384);
      mma_commit(&bars[B_C0]);
    }
  }
  __syncwarp();
  ok = mbar_wait(&bars[B_DKV], 0, 257) && ok;
  tc_fence_after();
  {
    float kr[16], ki[16], vr[16], vi[16];           // dk, dv
    tmem_ld16x2(tl + 128 + 16 * cq, kr, tl + 192 + 16 * cq, ki);
    tmem_ld16x2(tl + 384 + 16 * cq, vr, tl + 448 + 16 * cq, vi);
#pragma unroll
    for (int k = 0; k < K; ++k) cs[k] = (cp[k].x + cp[k].y) * ck[k];
    if (has_ds) {
      // a state's products run while the one before it is read: state k + 1 is issued once every warp has read what holds its
      // columns (dk and dv for state 1, state k - 1 after that)
#pragma unroll
      for (int k = 0; k < K; ++k) {
        if (k + 1 < K) {
          tc_fence_before();
          __syncthreads();
          if (issuer) {
            tc_fence_after();
            const uint32_t s1 = sl + ((k + 3) & 3) * 16384, c1 = tmem + 128 * ((k + 1) & 1);
            issue_state<true>(c1, v_r, s1);
            issue_state<false>(c1 + 256, k_r, s1);
            mma_commit(&bars[B_C1 + k]);
          }
          __syncwarp();
        }
        ok = mbar_wait(&bars[B_C0 + k], 0, 258) && ok;
        tc_fence_after();
        const uint32_t at = tl + 128 * (k & 1) + 16 * cq;
        const float e = __expf(fminf(0.f, tb.A[k * TC + TC - 1] - tb.A[k * TC + r]));
        float ur[16], ui[16];
        {
          float xr[16], xi[16];
          tmem_ld16x2(at, ur, at + 64, ui);
          row16(TK, r, cq, xr, xi);
          float2 d = make_float2(0.f, 0.f);
#pragma unroll
          for (int j = 0; j < 16; j += 2) {
            const float2 a = make_float2(ur[j], ur[j + 1]), b = make_float2(ui[j], ui[j + 1]);
            d = ffma2(make_float2(xr[j], xr[j + 1]), a, ffma2(make_float2(xi[j], xi[j + 1]), b, d));
            const float2 o = ffma2(make_float2(e, e), a, make_float2(kr[j], kr[j + 1])), p2 = ffma2(make_float2(e, e), b, make_float2(ki[j], ki[j + 1]));
            kr[j] = o.x; kr[j + 1] = o.y;
            ki[j] = p2.x; ki[j + 1] = p2.y;
          }
          cs[k] = fmaf(e, d.x + d.y, cs[k]);
        }
        tmem_ld16x2(at + 256, ur, at + 320, ui);
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          const float2 o = ffma2(make_float2(e, e), make_float2(ur[j], ur[j + 1]), make_float2(vr[j], vr[j + 1]));
          const float2 p2 = ffma2(make_float2(e, e), make_float2(ui[j], ui[j + 1]), make_float2(vi[j], vi[j + 1]));
          vr[j] = o.x; vr[j + 1] = o.y;
          vi[j] = p2.x; vi[j + 1] = p2.y;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < K; ++k) kdp[(cq * K + k) * TC + r] = cs[k];
    // q and dy have no reader left: their tiles take the rows of dk and dv
    put16(kr, ki, TQ, reinterpret_cast<__nv_bfloat16*>(p.dk) + obase, r, cq, len == TC, valid && ok);
    put16(vr, vi, TY, reinterpret_cast<__nv_bfloat16*>(p.dv) + obase, r, cq, len == TC, valid && ok);
  }
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc<512>(tmem);
  }
  if (lane == 0 && len == TC && ok) {
    if (warp < 8) store_box(&maps.dk, TQ, warp, row0);
    else store_box(&maps.dv, TY, warp - 8, row0);
  }

  // ---- dc, and the decay gradient: da_u = sum_{t >= u} (Re<q,dq> - Re<k,dk>)_t.  The raw values would accumulate their
  // errors as a random walk over the whole sequence, so the suffix sum is anchored at every chunk boundary with the value
  // the reverse carry left there (Re<dS, S>, fp32) and the small mismatch of the chunk is spread linearly over its tokens.
  float suffix = 0.f;
  if (ek < K) {
    float2 dc = make_float2(0.f, 0.f);
    float kd = 0.f;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const float2 a = dcp[(g * K + ek) * TC + et];
      dc.x += a.x;
      dc.y += a.y;
      kd += kdp[(g * K + ek) * TC + et];
    }
    if (p.dcoef != nullptr && et < len && ok) *reinterpret_cast<float2*>(p.dcoef + eg * 2) = dc;
    tb.row[ek * TC + et] = et < len ? c_e.x * dc.x + c_e.y * dc.y - kd : 0.f;
    if ((warp & 3) < 2) {
      double a2 = (double)an0 + (double)an1;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) a2 += __shfl_xor_sync(0xffffffffu, a2, o);
      if (lane == 0) anc[ek * 2 + (warp & 3)] = (float)a2;
    }
  }
  __syncthreads();
  if (ek < K) {
    suffix = tb.row[ek * TC + et_rev];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float n = __shfl_up_sync(0xffffffffu, suffix, o);
      if (lane >= o) suffix += n;
    }
    if (lane == 31) wsum[ek * 4 + (warp & 3)] = suffix;
  }
  __syncthreads();
  if (ek < K) {
    const int w = warp & 3;
    for (int i = 0; i < w; ++i) suffix += wsum[ek * 4 + i];
    const float total = wsum[ek * 4] + wsum[ek * 4 + 1] + wsum[ek * 4 + 2] + wsum[ek * 4 + 3];
    const float lo = anc[ek * 2], hi = anc[ek * 2 + 1], mismatch = total - (lo - hi);
    if (et_rev < len && ok) {
      const size_t gi = gamma_base(p, ek, L.b, h, L.t0 + et_rev);
      p.dgamma[gi] = (hi + suffix - mismatch * (float)(len - et_rev) / (float)len) / (g_e + p.eps);
    }
  }
  if (lane == 0) tma_store_wait_read();     // the staging blocks are read before this CTA's shared memory goes away
}

}  // namespace tcs
}  // namespace qpam
