// O(1)-per-token recurrent PAM step over a pool of per-sequence state slots.
//
// HBM-bound: per (sequence, head, state) the kernel streams a d x d complex matrix in and out
// once (2 * d*d*2*sizeof(state) bytes) for ~22 d^2 flops.  Each thread owns 16-byte pieces of
// state rows (128-bit coalesced loads/stores, a row is covered by consecutive lanes), all loads of
// a state are issued before the first use, and the read-out y = S q is finished with warp
// shuffles.  Continuous batching: `slot_ids` picks the slot of every live sequence, so sequences
// join and leave by editing that index vector only.
#include "common.cuh"
#include "elementwise.cuh"
#include "umma.cuh"

namespace qpam {

template <typename ST>
struct StateVec;
template <>
struct StateVec<float> {
  static constexpr int NC = 2;  // complex entries per 16-byte vector
  static __device__ __forceinline__ void load(const float* p, float2 (&o)[NC]) {
    const float4 v = __ldcs(reinterpret_cast<const float4*>(p));
    o[0] = make_float2(v.x, v.y);
    o[1] = make_float2(v.z, v.w);
  }
  static __device__ __forceinline__ void store(float* p, const float2 (&o)[NC]) {
    __stcs(reinterpret_cast<float4*>(p), make_float4(o[0].x, o[0].y, o[1].x, o[1].y));
  }
};
template <>
struct StateVec<__nv_bfloat16> {
  static constexpr int NC = 4;
  static __device__ __forceinline__ void load(const __nv_bfloat16* p, float2 (&o)[NC]) {
    const uint4 v = __ldcs(reinterpret_cast<const uint4*>(p));
    const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int i = 0; i < NC; ++i) o[i] = __bfloat1622float2(b[i]);
  }
  static __device__ __forceinline__ void store(__nv_bfloat16* p, const float2 (&o)[NC]) {
    uint4 v;
    __nv_bfloat162* b = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
    for (int i = 0; i < NC; ++i) b[i] = __float22bfloat162_rn(o[i]);
    __stcs(reinterpret_cast<uint4*>(p), v);
  }
};

struct DecodeParams {
  void* pool;
  const int32_t* slot_ids;
  const void *q, *k, *v;
  const float* gamma;  // [K,n,H]
  const float* coef;   // [K,n,H,2] or null
  void* y;
  int64_t n_slots;
  int32_t L, layer, n, H, K;
};

// grid = n*H CTAs; block = min(256, D*D/NC) threads.
template <int D, typename ST, typename T>
__global__ void __launch_bounds__(256) k_decode_step(DecodeParams p) {
  constexpr int NC = StateVec<ST>::NC;
  constexpr int LPR = D / NC;                                  // lanes per state row
  constexpr int NTH = (D * D / NC) < 256 ? (D * D / NC) : 256;  // threads
  constexpr int RPP = NTH / LPR;                               // rows per pass
  constexpr int PASSES = D / RPP;
  __shared__ float2 sq[D], sk[D], sv[D];
  const int tid = threadIdx.x;
  pdl_wait();
  const int seq = blockIdx.x / p.H, h = blockIdx.x - seq * p.H;
  const int slot = p.slot_ids[seq];
  const size_t vb = ((size_t)seq * p.H + h) * D * 2;
  if (slot < 0 || slot >= p.n_slots) {        // padded / retired entry: no state, but a defined output (see k_decode_step_bulk)
    for (int i = tid; i < D; i += NTH) IO<T>::st2(reinterpret_cast<T*>(p.y) + vb + 2 * i, make_float2(0.f, 0.f));
    return;
  }
  if (tid < D) {
    sq[tid] = IO<T>::ld2(reinterpret_cast<const T*>(p.q) + vb + 2 * tid);
    sk[tid] = IO<T>::ld2(reinterpret_cast<const T*>(p.k) + vb + 2 * tid);
    sv[tid] = IO<T>::ld2(reinterpret_cast<const T*>(p.v) + vb + 2 * tid);
  }
  __syncthreads();
  const int row0 = tid / LPR, j0 = (tid % LPR) * NC;
  float2 kq[NC], qq[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    kq[c] = sk[j0 + c];
    qq[c] = sq[j0 + c];
  }
  float2 yacc[PASSES];
#pragma unroll
  for (int r = 0; r < PASSES; ++r) yacc[r] = make_float2(0.f, 0.f);
  for (int k = 0; k < p.K; ++k) {
    ST* S = reinterpret_cast<ST*>(p.pool) +
            ((((size_t)slot * p.L + p.layer) * p.K + k) * p.H + h) * (size_t)(D * D * 2);
    const size_t gi = ((size_t)k * p.n + seq) * p.H + h;
    const float g = p.gamma[gi];
    float2 cf = make_float2(1.f, 0.f);
    if (p.coef != nullptr) cf = *reinterpret_cast<const float2*>(p.coef + gi * 2);
    float2 s[PASSES][NC];
#pragma unroll
    for (int r = 0; r < PASSES; ++r) StateVec<ST>::load(S + ((size_t)(row0 + r * RPP) * D + j0) * 2, s[r]);
#pragma unroll
    for (int r = 0; r < PASSES; ++r) {
      const float2 vi = sv[row0 + r * RPP];
      float2 part = make_float2(0.f, 0.f);
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const float2 o = cmulc(vi, kq[c]);  // v_i conj(k_j)
        s[r][c].x = fmaf(g, s[r][c].x, o.x);
        s[r][c].y = fmaf(g, s[r][c].y, o.y);
        cfma<false, false>(part, s[r][c], qq[c]);
      }
      StateVec<ST>::store(S + ((size_t)(row0 + r * RPP) * D + j0) * 2, s[r]);
      const float2 m = cmul(cf, part);
      yacc[r].x += m.x;
      yacc[r].y += m.y;
    }
  }
#pragma unroll
  for (int r = 0; r < PASSES; ++r) {
    float2 a = yacc[r];
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) {
      a.x += __shfl_xor_sync(0xffffffffu, a.x, o);
      a.y += __shfl_xor_sync(0xffffffffu, a.y, o);
    }
    if ((tid % LPR) == 0) IO<T>::st2(reinterpret_cast<T*>(p.y) + vb + 2 * (row0 + r * RPP), a);
  }
}

// ------------------------------------------------------------------------------------------------
// bf16 state, d = 64: the K states of one (sequence, head) are 16 KB each.  They are brought into
// shared memory by bulk copies issued up front by one thread (all K in flight at once, independent of
// the register file), updated in place there, and written back by bulk copies.  With ~50 KB per CTA
// four CTAs fit on an SM, i.e. ~190 KB of loads in flight per SM.
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ void bulk_load(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               :
               : "r"(umma::smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(gsrc)), "r"(bytes), "r"(umma::smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void bulk_store(void* gdst, const void* smem_src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
               :
               : "l"(reinterpret_cast<uint64_t>(gdst)), "r"(umma::smem_u32(smem_src)), "r"(bytes)
               : "memory");
}

constexpr int DEC_BULK_STATE_BYTES = 64 * 64 * 2 * 2;  // one bf16 state

// q, k, v, decay and read-out weights of one token and head, from the outputs of the layer's input projections: what k_pam_front
// writes for the whole batch, formed here by the CTA that uses it while its states are on their way.  The gates that read |x| (one
// to ten rows of D for a head) are products of this CTA too, a warp each.  Two launches less a layer where there are such gates, one
// where not: a step of the 12-layer model with three states, 128 / 48 / 20 sequences: 1010 -> 966, 773 -> 716, 688 -> 629 us; with one
// state, 256 / 20: 938 -> 939, 598 -> 581 (256: bound by the states, and k_pam_front ran beside their first loads).
struct FrontOut {
  float2 q[64], k[64], v[64];
  float gate[2 + 2 * QPAM_MAX_STATES];      // dt | protect | phases | scores
  float gamma[QPAM_MAX_STATES];
  float2 coef[QPAM_MAX_STATES];
};
__device__ __forceinline__ void decode_front(const qpam_decode_front_args& a, int seq, int h, FrontOut& o) {
  typedef __nv_bfloat16 bf16;
  const qpam_front_args& f = a.f;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, K = f.K;
  float2 x[3], rot = make_float2(1.f, 0.f);
  if (tid < 64) {
    const bf16* src = reinterpret_cast<const bf16*>(f.qkv) + (int64_t)seq * f.ld_qkv + (h * 64 + tid) * 2;
#pragma unroll
    for (int w = 0; w < 3; ++w) x[w] = IO<bf16>::ld2(src + (int64_t)w * f.H * 128);
    if (f.rope) {
      int64_t pos = f.positions ? f.positions[seq] : f.offset;
      pos = pos < 0 ? 0 : (pos >= f.rope_len ? f.rope_len - 1 : pos);
      rot = *reinterpret_cast<const float2*>(f.rope + (pos * 64 + tid) * 2);
    }
  } else {
    for (int i = warp - 2; i < 2 + 2 * K; i += 6) {
      const int what = i < 2 ? i : i < 2 + K ? 2 : 3, at = what < 2 ? h : h * K + (i - 2) % K;
      const void* raw = what == 0 ? f.dt : what == 1 ? f.pg : what == 2 ? f.phase : f.score;
      const int64_t ld = what == 0 ? f.ld_dt : what == 1 ? f.ld_pg : what == 2 ? f.ld_phase : f.ld_score;
      float v = 0.f;
      if (raw) {
        v = __bfloat162float(reinterpret_cast<const bf16*>(raw)[seq * ld + at]);
      } else if (a.mag_row[what] >= 0) {
        const int row = a.mag_row[what] + at;
        const uint4* m = reinterpret_cast<const uint4*>(reinterpret_cast<const bf16*>(a.mag) + (int64_t)seq * a.D);
        const uint4* w = reinterpret_cast<const uint4*>(reinterpret_cast<const bf16*>(a.w_mag) + (int64_t)row * a.D);
        for (int g = lane; g < a.D / 8; g += 32) {
          const uint4 p = m[g], r = w[g];
          const uint32_t pw[4] = {p.x, p.y, p.z, p.w}, rw[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            v = fmaf(__uint_as_float(pw[e] << 16), __uint_as_float(rw[e] << 16), v);
            v = fmaf(__uint_as_float(pw[e] & 0xffff0000u), __uint_as_float(rw[e] & 0xffff0000u), v);
          }
        }
        v = ew::warp_sum(v) + __bfloat162float(reinterpret_cast<const bf16*>(a.b_mag)[row]);
        v = __bfloat162float(__float2bfloat16_rn(v));
      }
      if (lane == 0) o.gate[i] = v;
    }
  }
  __syncthreads();
  const bool has_pg = f.pg != nullptr || a.mag_row[1] >= 0, has_phase = f.phase != nullptr || a.mag_row[2] >= 0, has_score = f.score != nullptr || a.mag_row[3] >= 0;
  const float prot = has_pg ? ew::sigmoidf_(o.gate[1]) : 0.f;
  if (tid < 64) {
    auto store = [&](float2& at, float re, float im) { at = __bfloat1622float2(__floats2bfloat162_rn(re, im)); };      // (as they are stored otherwise)
    store(o.q[tid], (x[0].x * rot.x - x[0].y * rot.y) * f.q_scale, (x[0].x * rot.y + x[0].y * rot.x) * f.q_scale);
    store(o.k[tid], x[1].x * rot.x - x[1].y * rot.y, x[1].x * rot.y + x[1].y * rot.x);
    const float keep = 1.f - prot;
    store(o.v[tid], x[2].x * keep, x[2].y * keep);
  } else if (tid < 64 + K) {
    const int k = tid - 64;
    float base = ew::sigmoidf_(-(o.gate[0] + f.dt_bias[h] + (f.state_dt_offset ? f.state_dt_offset[k] : 0.f)));      // exp(-softplus(x))
    if (f.gamma_floor > 0.f) base = f.gamma_floor + (1.f - f.gamma_floor) * base;
    o.gamma[k] = base * (1.f - prot) + prot;
    float w = 1.f, sn = 0.f, cs = 1.f;
    if (K > 1) {
      if (has_score) {
        const float* s = o.gate + 2 + K;
        float top = -INFINITY, sum = 0.f;
        for (int i = 0; i < K; ++i) top = fmaxf(top, s[i]);
        for (int i = 0; i < K; ++i) sum += __expf(s[i] - top);
        w = __expf(s[k] - top) / sum * (float)K;
      }
      if (has_phase) sincosf(o.gate[2 + k], &sn, &cs);
    }
    o.coef[k] = make_float2(w * cs, w * sn);
  }
  __syncthreads();
}

// FRONT: q, k, v, gamma and coef come from `decode_front` instead of memory.
template <typename T, bool FRONT>
__global__ void __launch_bounds__(256) k_decode_step_bulk(DecodeParams p, const __grid_constant__ qpam_decode_front_args front) {
  constexpr int D = 64, NC = 4, LPR = D / NC, RPP = 256 / LPR, PASSES = D / RPP;
  extern __shared__ __align__(128) unsigned char dec_smem[];
  __shared__ FrontOut in;
  __shared__ __align__(8) uint64_t bar[QPAM_MAX_STATES];   // one per state: work on state k starts when it has landed
  const int tid = threadIdx.x;
  const int seq = blockIdx.x / p.H, h = blockIdx.x - seq * p.H;
  const size_t state_elems = (size_t)D * D * 2;
  __nv_bfloat16* pool = reinterpret_cast<__nv_bfloat16*>(p.pool);
  // While the predecessor (the kernel that forms q, k, v) ends, the states are asked into L2.  Nothing is read: should something
  // still write the slot or its index, it is the wait that orders the loads behind it.
  if (tid < p.K) {
    const int hint = __ldcg(p.slot_ids + seq);
    if (hint >= 0 && hint < p.n_slots)
      umma::bulk_prefetch_l2(pool + ((((size_t)hint * p.L + p.layer) * p.K + tid) * p.H + h) * state_elems, DEC_BULK_STATE_BYTES);
  }
  pdl_wait();
  const int slot = __ldcg(p.slot_ids + seq);
  const size_t vb = ((size_t)seq * p.H + h) * D * 2;
  if (slot < 0 || slot >= p.n_slots) {        // padded / retired entry (whole CTA): no state, but a defined output -- the row goes on
    if (tid < D) IO<T>::st2(reinterpret_cast<T*>(p.y) + vb + 2 * tid, make_float2(0.f, 0.f));      // through the step to an id
    return;
  }
  const size_t base = (((size_t)slot * p.L + p.layer) * p.K) * p.H + h;  // + k * H per state
  if (tid == 0) {
    for (int k = 0; k < p.K; ++k) umma::mbar_init(&bar[k], 1);
    umma::fence_barrier_init();
    for (int k = 0; k < p.K; ++k) {
      umma::mbar_arrive_expect_tx(&bar[k], (uint32_t)DEC_BULK_STATE_BYTES);
      bulk_load(dec_smem + (size_t)k * DEC_BULK_STATE_BYTES, pool + (base + (size_t)k * p.H) * state_elems,
                DEC_BULK_STATE_BYTES, &bar[k]);
    }
  }
  if constexpr (FRONT) {
    decode_front(front, seq, h, in);
  } else {
    if (tid < D) {
      in.q[tid] = IO<T>::ld2(reinterpret_cast<const T*>(p.q) + vb + 2 * tid);
      in.k[tid] = IO<T>::ld2(reinterpret_cast<const T*>(p.k) + vb + 2 * tid);
      in.v[tid] = IO<T>::ld2(reinterpret_cast<const T*>(p.v) + vb + 2 * tid);
    }
    __syncthreads();  // (here as in decode_front: it also publishes the barriers' initialisation to the waiters)
  }
  bool arrived = true;
  const int row0 = tid / LPR, j0 = (tid % LPR) * NC;
  float2 kq[NC], qq[NC], yacc[PASSES];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    kq[c] = in.k[j0 + c];
    qq[c] = in.q[j0 + c];
  }
#pragma unroll
  for (int r = 0; r < PASSES; ++r) yacc[r] = make_float2(0.f, 0.f);
  {
    for (int k = 0; k < p.K; ++k) {
      // on a give-up the error word is set and the arithmetic below is skipped; the barriers are not
      arrived = umma::mbar_wait(&bar[k], 0, 31) && arrived;
      __nv_bfloat16* S = reinterpret_cast<__nv_bfloat16*>(dec_smem + (size_t)k * DEC_BULK_STATE_BYTES);
      const size_t gi = ((size_t)k * p.n + seq) * p.H + h;
      const float g = FRONT ? in.gamma[k] : p.gamma[gi];
      float2 cf = make_float2(1.f, 0.f);
      if (FRONT) cf = in.coef[k];
      else if (p.coef != nullptr) cf = *reinterpret_cast<const float2*>(p.coef + gi * 2);
#pragma unroll
      for (int r = 0; r < PASSES; ++r) {
        if (!arrived) break;
        const int row = row0 + r * RPP;
        uint4* cell = reinterpret_cast<uint4*>(S + ((size_t)row * D + j0) * 2);
        uint4 raw = *cell;
        __nv_bfloat162* b = reinterpret_cast<__nv_bfloat162*>(&raw);
        const float2 vi = in.v[row];
        float2 part = make_float2(0.f, 0.f);
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          float2 e = __bfloat1622float2(b[c]);
          const float2 o = cmulc(vi, kq[c]);  // v_i conj(k_j)
          e.x = fmaf(g, e.x, o.x);
          e.y = fmaf(g, e.y, o.y);
          cfma<false, false>(part, e, qq[c]);
          b[c] = __float22bfloat162_rn(e);
        }
        *cell = raw;
        const float2 m = cmul(cf, part);
        yacc[r].x += m.x;
        yacc[r].y += m.y;
      }
      umma::fence_proxy_async();  // the bulk store below reads what the generic proxy just wrote
      __syncthreads();
      if (tid == 0 && arrived) {    // state k goes back while state k+1 is being updated
        bulk_store(pool + (base + (size_t)k * p.H) * state_elems, dec_smem + (size_t)k * DEC_BULK_STATE_BYTES,
                   DEC_BULK_STATE_BYTES);
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      }
    }
  }
  if (tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // shared memory must outlive the copies
#pragma unroll
  for (int r = 0; r < PASSES; ++r) {
    float2 a = yacc[r];
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) {
      a.x += __shfl_xor_sync(0xffffffffu, a.x, o);
      a.y += __shfl_xor_sync(0xffffffffu, a.y, o);
    }
    if ((tid % LPR) == 0) IO<T>::st2(reinterpret_cast<T*>(p.y) + vb + 2 * (row0 + r * RPP), a);
  }
}

template <typename T, bool FRONT = false>
static int launch_decode_bulk(const DecodeParams& p, cudaStream_t st, const qpam_decode_front_args& front = {}) {
  const size_t smem = (size_t)p.K * DEC_BULK_STATE_BYTES;
  auto kern = k_decode_step_bulk<T, FRONT>;
  const int rc = allow_smem(reinterpret_cast<const void*>(kern), smem);
  if (rc) return rc;
  launch_after(kern, p.n * p.H, 256, smem, st, p, front);
  QPAM_LAUNCH_CHECK("k_decode_step_bulk");
  return QPAM_OK;
}

int decode_device_status(int* value, bool clear) {
  QPAM_CUDA(umma::read_device_error(value, clear));
  return QPAM_OK;
}

template <int D, typename ST, typename T>
static int launch_decode(const DecodeParams& p, cudaStream_t st) {
  constexpr int NC = StateVec<ST>::NC;
  constexpr int NTH = (D * D / NC) < 256 ? (D * D / NC) : 256;
  launch_after(k_decode_step<D, ST, T>, p.n * p.H, NTH, 0, st, p);
  QPAM_LAUNCH_CHECK("k_decode_step");
  return QPAM_OK;
}

template <typename ST>
__global__ void k_pool_store(ST* pool, const int32_t* slot_ids, const float* states, int64_t n_slots, int L,
                             int layer, int S, int H, int K, int dd2) {
  // one CTA per (k, s, h); states [K,S,H,dd2] -> pool[slot, layer, k, h, dd2]
  const int h = blockIdx.x % H, s = (blockIdx.x / H) % S, k = blockIdx.x / (H * S);
  const int slot = slot_ids[s];
  if (slot < 0 || slot >= n_slots) return;
  const float* src = states + (((size_t)k * S + s) * H + h) * dd2;
  ST* dst = pool + ((((size_t)slot * L + layer) * K + k) * H + h) * (size_t)dd2;
  for (int e = threadIdx.x; e < dd2; e += blockDim.x) IO<ST>::st(dst + e, src[e]);
}

}  // namespace qpam

using namespace qpam;

extern "C" int qpam_decode_step(void* state_pool, int32_t state_dtype, int64_t n_slots, int32_t L,
                                int32_t layer, const int32_t* slot_ids, const void* q, const void* k,
                                const void* v, const float* gamma, const float* coef, void* y, int32_t n,
                                int32_t H, int32_t d, int32_t K, int32_t io_dtype, void* stream) {
  QPAM_REQUIRE(state_pool && slot_ids && q && k && v && gamma && y, "decode: NULL pointer argument");
  QPAM_REQUIRE(d == 16 || d == 32 || d == 64, "decode: head dim d=%d not in {16,32,64}", d);
  QPAM_REQUIRE(K >= 1 && K <= QPAM_MAX_STATES, "decode: K=%d outside [1,%d]", K, QPAM_MAX_STATES);
  QPAM_REQUIRE(n >= 0 && H >= 1 && L >= 1 && layer >= 0 && layer < L, "decode: bad n/H/L/layer");
  QPAM_REQUIRE(state_dtype == QPAM_F32 || state_dtype == QPAM_BF16, "decode: state_dtype %d unknown", state_dtype);
  QPAM_REQUIRE(io_dtype == QPAM_F32 || io_dtype == QPAM_BF16, "decode: io_dtype %d unknown", io_dtype);
  QPAM_REQUIRE(((uintptr_t)state_pool & 15) == 0, "decode: state_pool must be 16-byte aligned");
  if (n == 0) return QPAM_OK;
  DecodeParams p{state_pool, slot_ids, q, k, v, gamma, coef, y, n_slots, L, layer, n, H, K};
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (d == 64 && state_dtype == QPAM_BF16)   // shared-memory staged variant (bulk copies)
    return io_dtype == QPAM_F32 ? launch_decode_bulk<float>(p, st) : launch_decode_bulk<__nv_bfloat16>(p, st);
#define QPAM_DEC(DD)                                                                          \
  if (state_dtype == QPAM_F32)                                                                \
    return io_dtype == QPAM_F32 ? launch_decode<DD, float, float>(p, st)                      \
                                : launch_decode<DD, float, __nv_bfloat16>(p, st);             \
  return io_dtype == QPAM_F32 ? launch_decode<DD, __nv_bfloat16, float>(p, st)                \
                              : launch_decode<DD, __nv_bfloat16, __nv_bfloat16>(p, st);
  if (d == 16) { QPAM_DEC(16) }
  if (d == 32) { QPAM_DEC(32) }
  QPAM_DEC(64)
#undef QPAM_DEC
}

extern "C" int qpam_decode_front(void* state_pool, int64_t n_slots, int32_t L, int32_t layer, const int32_t* slot_ids,
                                 const qpam_decode_front_args* a, void* y, int32_t n, void* stream) {
  QPAM_REQUIRE(state_pool && slot_ids && a && y && a->f.qkv && a->f.dt_bias, "decode front: NULL pointer argument");
  const qpam_front_args& f = a->f;
  QPAM_REQUIRE(f.d == 64 && f.io_dtype == QPAM_BF16, "decode front: offered for bf16 and head dim 64");
  QPAM_REQUIRE(f.K >= 1 && f.K <= QPAM_MAX_STATES && f.H >= 1, "decode front: bad H/K = %d/%d", f.H, f.K);
  QPAM_REQUIRE(n >= 0 && L >= 1 && layer >= 0 && layer < L, "decode front: bad n/L/layer");
  QPAM_REQUIRE(((uintptr_t)state_pool & 15) == 0 && (((uintptr_t)f.qkv | (uintptr_t)y) & 3) == 0 && f.ld_qkv % 2 == 0, "decode front: unaligned pointer");
  QPAM_REQUIRE(f.dt != nullptr || a->mag_row[0] >= 0, "decode front: no decay projection");
  QPAM_REQUIRE(!f.rope || f.rope_len > 0, "decode front: empty rotary table");
  bool from_mag = false;
  for (int i = 0; i < 4; ++i) from_mag = from_mag || a->mag_row[i] >= 0;
  QPAM_REQUIRE(!from_mag || (a->mag && a->w_mag && a->b_mag && a->D >= 8 && a->D % 8 == 0 && (((uintptr_t)a->mag | (uintptr_t)a->w_mag) & 15) == 0),
               "decode front: gates of |x| need mag, w_mag (16-byte aligned rows) and b_mag");
  if (n == 0) return QPAM_OK;
  const DecodeParams p{state_pool, slot_ids, nullptr, nullptr, nullptr, nullptr, nullptr, y, n_slots, L, layer, n, f.H, f.K};
  return launch_decode_bulk<__nv_bfloat16, true>(p, reinterpret_cast<cudaStream_t>(stream), *a);
}

extern "C" int qpam_pool_store(void* state_pool, int32_t state_dtype, int64_t n_slots, int32_t L,
                               int32_t layer, const int32_t* slot_ids, const float* states, int32_t S,
                               int32_t H, int32_t d, int32_t K, void* stream) {
  QPAM_REQUIRE(state_pool && slot_ids && states, "pool_store: NULL pointer argument");
  QPAM_REQUIRE(S >= 0 && H >= 1 && K >= 1 && d >= 1 && L >= 1 && layer >= 0 && layer < L, "pool_store: bad sizes");
  QPAM_REQUIRE(state_dtype == QPAM_F32 || state_dtype == QPAM_BF16, "pool_store: state_dtype %d unknown", state_dtype);
  if (S == 0) return QPAM_OK;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int dd2 = d * d * 2;
  if (state_dtype == QPAM_F32)
    k_pool_store<float><<<K * S * H, 256, 0, st>>>(reinterpret_cast<float*>(state_pool), slot_ids, states, n_slots, L, layer, S, H, K, dd2);
  else
    k_pool_store<__nv_bfloat16><<<K * S * H, 256, 0, st>>>(reinterpret_cast<__nv_bfloat16*>(state_pool), slot_ids, states, n_slots, L, layer, S, H, K, dd2);
  QPAM_LAUNCH_CHECK("k_pool_store");
  return QPAM_OK;
}
