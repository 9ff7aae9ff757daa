// One decode step of a whole model for a handful of sequences (n <= 16), from token ids to the next ids or logits.
//
// What bounds it: every weight is used for n rows only, so the step is the time to stream the weights once (0.06 ms of
// HBM for the 12-block dim-768 model, plus 0.02 ms for the tied head) and the latency of its chain of dependent phases,
// five per block.  Three things bring it towards that:
//   * half the weight bytes.  A complex projection is packed as a real matrix [2*out, 2*in] whose rows (o, re) =
//     (Wr, -Wi) and (o, im) = (Wi, Wr) hold the same numbers, so only the even rows are read here: with x = (xr, xi) the
//     row gives the real part, with the rotated x' = (xi, -xr) the imaginary part.  Both are columns of one product.
//   * five phases instead of ~13 launches per block.  Residual add and norm sit in front of the projection that reads
//     them, the gated unit and the rotary rotation behind theirs, the gate arithmetic in the recurrent step.
//   * weights requested ahead of the dependency.  n <= 4: one persistent kernel whose CTAs request the next phase's weights
//     between arriving at a grid barrier and waiting for it.  n <= 16: a kernel per phase with programmatic dependent
//     launch, each requesting its first weights before it waits for its predecessor.
// The product is mma.sync m16n8k16 with 16 weight rows as A straight from global memory (16-byte loads, no shared memory)
// and the sequences as the 8 columns: tcgen05 would need its 128-row tiles staged through shared memory for the same
// bytes, and they would give the D-row projections 12 CTAs.
// Step of that model, replayed from a graph, K = 3 states (library GEMMs on the packed matrices, ~160 launches, before):
// n = 1 760 -> 267 us, n = 4 780 -> 329 us, n = 8 -> 448 us, n = 16 820 -> 516 us; at n = 32 the library route is as fast.
#include <cooperative_groups.h>

#include "common.cuh"
#include "elementwise.cuh"
#include "umma.cuh"

namespace qpam {
namespace {
using namespace ew;
typedef __nv_bfloat16 bf16;

constexpr int ST_WARPS = 8;
constexpr int ST_THREADS = ST_WARPS * 32;
constexpr int ST_PF = 6;             // 32-wide K blocks of weights requested ahead per warp (48 registers)
constexpr int ST_ONE_N = 4;          // up to this many sequences the step is one persistent kernel
constexpr int ST_ONE_LAYERS = 64;    // (its layer pointers are kernel parameters)

__device__ __forceinline__ uint4 ld_weight(const bf16* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// (re, im) -> (im, -re)
__device__ __forceinline__ uint32_t rot(uint32_t w) { return __byte_perm(w, w, 0x1032) ^ 0x80000000u; }
__device__ __forceinline__ float rbf(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// 4 complex values another CTA of this kernel wrote: not through L1
__device__ __forceinline__ void ldcg4(const bf16* p, float (&r)[4], float (&i)[4]) {
  const uint4 u = __ldcg(reinterpret_cast<const uint4*>(p));
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    r[j] = __uint_as_float(w[j] << 16);
    i[j] = __uint_as_float(w[j] & 0xffff0000u);
  }
}

enum { EPI_GATE, EPI_COMPLEX, EPI_FRONT, EPI_VOCAB };

struct Skinny {
  // operand
  const bf16* x;            // [n, K] input rows
  // weights
  const bf16* w;
  const bf16* w2;           // EPI_FRONT: the rows that read |xn|
  int64_t ld;
  int32_t n, K, rows;       // K scalars per row of w; rows: complex outputs (EPI_VOCAB: real ones)
  int32_t rows_a, rows_m;   // EPI_FRONT: real rows behind the complex ones, and rows of w2
  // epilogue
  const bf16* bias;         // EPI_COMPLEX: [2*rows] or null; EPI_FRONT: bias of the rows_a rows
  const bf16* bias2;        // EPI_FRONT: bias of the rows_m rows
  void* out;
  const float* act_bias;    // EPI_GATE
  const float* act_beta;
  bf16 *q, *k, *v;          // EPI_FRONT
  float* gates;             // EPI_FRONT: [n, rows_a + rows_m]
  const float* rope;
  const int64_t* positions;
  int64_t rope_len;
  int32_t H, d;
  float q_scale;
  unsigned long long* best; // EPI_VOCAB: running arg-max per sequence, or
  bf16* logits;             //            logits [n, ld_logits]
  int64_t ld_logits;
  int64_t* next_ids;
  unsigned int* done;
};

__device__ __forceinline__ unsigned long long best_key(float v, int idx) {
  const uint32_t u = __float_as_uint(v);
  const uint32_t k = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
  return ((unsigned long long)k << 32) | (uint32_t)~idx;      // the largest value, the lowest index among equals
}

// Input rows into shared memory (row stride xs_ld scalars); PLANAR: interleaved -> [re | im].
template <bool PLANAR>
__device__ __forceinline__ void load_rows(const Skinny& p, bf16* xs, int xs_ld, int k0, int k1) {
  const int vec = (k1 - k0) >> 3;
  for (int i = threadIdx.x; i < p.n * vec; i += ST_THREADS) {
    const int r = i / vec, g = i - r * vec;
    const uint4 u = *reinterpret_cast<const uint4*>(p.x + (int64_t)r * p.K + k0 + g * 8);
    if (PLANAR) {
      const uint32_t w[4] = {u.x, u.y, u.z, u.w};
      const int j = g * 4;
      *reinterpret_cast<uint2*>(xs + (size_t)r * xs_ld + j) = make_uint2(__byte_perm(w[0], w[1], 0x5410), __byte_perm(w[2], w[3], 0x5410));
      *reinterpret_cast<uint2*>(xs + (size_t)r * xs_ld + (p.K >> 1) + j) = make_uint2(__byte_perm(w[0], w[1], 0x7632), __byte_perm(w[2], w[3], 0x7632));
    } else {
      *reinterpret_cast<uint4*>(xs + (size_t)r * xs_ld + g * 8) = u;
    }
  }
}

// Row stride of the input rows in shared memory, in scalars: 64 bytes off a multiple of 128, so that the eight rows (or
// four) of a B fragment start in different banks.
__host__ __device__ inline int row_ld(int kblocks) { return kblocks * 32 + ((kblocks & 1) ? 0 : 32); }

// acc += A * B over one 32-wide K block.  The lane's 16 bytes of a weight row are k = 8c .. 8c+7 (c = lane & 3); the order
// of k inside the block does not matter as long as both operands use the same one.
template <int NT, bool ROT>
__device__ __forceinline__ void block_mma(float (&acc)[NT][4], const uint4& lo, const uint4& hi, const bf16* xs, int xs_ld, int k, int lane) {
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    const int col = lane >> 2;
    const int seq = ROT ? t * 4 + (col >> 1) : t * 8 + col;
    uint4 b = *reinterpret_cast<const uint4*>(xs + (size_t)seq * xs_ld + k + (lane & 3) * 8);
    if (ROT && (col & 1)) { b.x = rot(b.x); b.y = rot(b.y); b.z = rot(b.z); b.w = rot(b.w); }
    mma16816(acc[t], lo.x, hi.x, lo.y, hi.y, b.x, b.y);
    mma16816(acc[t], lo.z, hi.z, lo.w, hi.w, b.z, b.w);
  }
}

// A CTA forms 16 output rows; its 8 warps split K (interleaved 32-wide blocks), a cluster of CTAs splits it further when
// a projection has few rows.  NT: groups of four sequences.
template <int NT, int EPI>
__global__ void __launch_bounds__(ST_THREADS, NT <= 2 ? 3 : 2) k_step_proj(Skinny p) {
  extern __shared__ __align__(16) unsigned char smem[];
  namespace cg = cooperative_groups;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int cs = EPI == EPI_COMPLEX ? (int)cg::this_cluster().num_blocks() : 1;
  const int rank = EPI == EPI_COMPLEX ? (int)cg::this_cluster().block_rank() : 0;
  const int tile = (int)blockIdx.x / cs;
  const int kb_slice = ((p.K >> 5) + cs - 1) / cs;  // K blocks of this CTA of the cluster
  const int xs_ld = row_ld(kb_slice);
  bf16* xs = reinterpret_cast<bf16*>(smem);
  float4* red = reinterpret_cast<float4*>(smem + (size_t)NT * 4 * xs_ld * sizeof(bf16));
  pdl_trigger();

  // ---- the two weight rows of this lane, and which kind of tile this is
  const int nq = EPI == EPI_FRONT ? p.rows / 16 : 0;
  const int na = EPI == EPI_FRONT ? (p.rows_a + 15) / 16 : 0;
  const bool is_mag = EPI == EPI_FRONT && tile >= nq + na;
  const bool is_real = EPI == EPI_FRONT && tile >= nq;
  const int r0 = lane >> 2;
  const bf16 *wl, *wh;
  if (EPI == EPI_GATE) {                            // 8 gate rows and the 8 up rows of the same channels
    wl = p.w + (int64_t)2 * (tile * 8 + r0) * p.ld;
    wh = p.w + (int64_t)2 * (p.rows + tile * 8 + r0) * p.ld;
  } else if (is_mag) {
    const int t = (tile - nq - na) * 16;
    wl = p.w2 + (int64_t)min(t + r0, p.rows_m - 1) * (p.K >> 1);
    wh = p.w2 + (int64_t)min(t + r0 + 8, p.rows_m - 1) * (p.K >> 1);
  } else if (is_real) {
    const int t = (tile - nq) * 16;
    wl = p.w + (int64_t)(2 * p.rows + min(t + r0, p.rows_a - 1)) * p.ld;
    wh = p.w + (int64_t)(2 * p.rows + min(t + r0 + 8, p.rows_a - 1)) * p.ld;
  } else {
    wl = p.w + (int64_t)2 * (tile * 16 + r0) * p.ld;
    wh = p.w + (int64_t)2 * (tile * 16 + r0 + 8) * p.ld;
  }
  const int Kt = is_mag ? p.K >> 1 : p.K;
  const int kb_all = Kt >> 5;
  const int b0 = rank * kb_slice, b1 = min(kb_all, b0 + kb_slice);
  const int x0 = b0 * 32;                // first scalar of the rows that shared memory holds
  const int off = (lane & 3) * 8;
  uint4 lo[ST_PF], hi[ST_PF];
#pragma unroll
  for (int i = 0; i < ST_PF; ++i) {
    const int b = b0 + warp + i * ST_WARPS;
    if (b < b1) {
      lo[i] = ld_weight(wl + b * 32 + off);
      hi[i] = ld_weight(wh + b * 32 + off);
    }
  }
  pdl_wait();

  load_rows<false>(p, xs, xs_ld, x0, EPI == EPI_COMPLEX ? b1 * 32 : p.K);
  __syncthreads();
  if (is_mag) {                                     // |xn| of the rounded rows, packed in front of itself row by row
    const int D = p.K >> 1;
    constexpr int MG = 4;                           // K <= 8 * 256 * MG / 2 is checked on the host
    for (int r = 0; r < p.n; ++r) {
      uint2 h[MG];
#pragma unroll
      for (int c = 0; c < MG; ++c) {
        const int g = tid + c * ST_THREADS;
        if (g * 4 < D) {
          float re[4], im[4];
          V4<bf16>::ld(xs + (size_t)r * xs_ld + g * 8, re, im);
#pragma unroll
          for (int j = 0; j < 4; ++j) re[j] = fsqrt_(re[j] * re[j] + im[j] * im[j] + MAG_EPS);
          h[c] = make_uint2(pack2(re[0], re[1]), pack2(re[2], re[3]));
        }
      }
      __syncthreads();
#pragma unroll
      for (int c = 0; c < MG; ++c) {
        const int g = tid + c * ST_THREADS;
        if (g * 4 < D) *reinterpret_cast<uint2*>(xs + (size_t)r * xs_ld + g * 4) = h[c];
      }
    }
    __syncthreads();
  }

  float acc[NT][4];
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[t][j] = 0.f;
  for (int b = b0 + warp; b < b1; b += ST_PF * ST_WARPS) {
#pragma unroll
    for (int i = 0; i < ST_PF; ++i) {
      const int bi = b + i * ST_WARPS;
      if (bi < b1) {
        block_mma<NT, true>(acc, lo[i], hi[i], xs, xs_ld, bi * 32 - x0, lane);
        const int bn = bi + ST_PF * ST_WARPS;
        if (bn < b1) {
          lo[i] = ld_weight(wl + bn * 32 + off);
          hi[i] = ld_weight(wh + bn * 32 + off);
        }
      }
    }
  }
#pragma unroll
  for (int t = 0; t < NT; ++t) red[(warp * NT + t) * 32 + lane] = make_float4(acc[t][0], acc[t][1], acc[t][2], acc[t][3]);
  __syncthreads();
  float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
  const bool mine = tid < NT * 32;
  if (mine) {
#pragma unroll
    for (int w = 0; w < ST_WARPS; ++w) {
      const float4 o = red[w * NT * 32 + tid];
      sum.x += o.x; sum.y += o.y; sum.z += o.z; sum.w += o.w;
    }
  }
  if (EPI == EPI_COMPLEX && cs > 1) {
    if (mine) red[tid] = sum;                       // (each thread overwrites only what it alone read)
    cg::this_cluster().sync();
    if (rank == 0 && mine) {
      for (int c = 1; c < cs; ++c) {
        const float4 o = *cg::this_cluster().map_shared_rank(&red[tid], c);
        sum.x += o.x; sum.y += o.y; sum.z += o.z; sum.w += o.w;
      }
    }
    cg::this_cluster().sync();
    if (rank != 0) return;
  }
  if (!mine) return;
  const int seq = (tid >> 5) * 4 + (lane & 3);      // (x, y) = (re, im) of row r0, (z, w) of row r0 + 8
  if (seq >= p.n) return;
  if (EPI == EPI_GATE) {
    const int ch = tile * 8 + r0;
    const float gr = rbf(sum.x), gi = rbf(sum.y), ur = rbf(sum.z), ui = rbf(sum.w);
    const MagInv um = mag_inv(ur * ur + ui * ui + MAG_EPS), gm = mag_inv(gr * gr + gi * gi + MAG_EPS);
    const float act = p.act_beta ? um.mag * sigmoidf_(p.act_beta[ch] * um.mag + p.act_bias[ch]) : fmaxf(um.mag + p.act_bias[ch], 0.f);
    const float h = sigmoidf_(gm.mag) * gm.inv * act * um.inv;
    reinterpret_cast<uint32_t*>(p.out)[(int64_t)seq * p.rows + ch] = pack2((gr * ur - gi * ui) * h, (gr * ui + gi * ur) * h);
  } else if (EPI == EPI_COMPLEX) {
    const int r = tile * 16 + r0;
    if (p.bias) {
      const __nv_bfloat162 *bb = reinterpret_cast<const __nv_bfloat162*>(p.bias);
      const float2 ba = __bfloat1622float2(bb[r]), bc = __bfloat1622float2(bb[r + 8]);
      sum.x += ba.x; sum.y += ba.y; sum.z += bc.x; sum.w += bc.y;
    }
    uint32_t* o = reinterpret_cast<uint32_t*>(p.out) + (int64_t)seq * p.rows;
    o[r] = pack2(sum.x, sum.y);
    o[r + 8] = pack2(sum.z, sum.w);
  } else if (!is_real) {                            // EPI_FRONT: q, k, v
    const int inner = p.H * p.d;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int r = tile * 16 + r0 + 8 * u;
      float re = u ? sum.z : sum.x, im = u ? sum.w : sum.y;
      const int which = r / inner, hj = r - which * inner;
      if (which < 2 && p.rope) {
        int64_t pos = p.positions[seq];
        pos = pos < 0 ? 0 : (pos >= p.rope_len ? p.rope_len - 1 : pos);
        const float2 cs_ = *reinterpret_cast<const float2*>(p.rope + (pos * p.d + hj % p.d) * 2);
        const float a = re * cs_.x - im * cs_.y;
        im = re * cs_.y + im * cs_.x;
        re = a;
      }
      const float m = which == 0 ? p.q_scale : 1.f;
      bf16* dst = which == 0 ? p.q : which == 1 ? p.k : p.v;
      reinterpret_cast<uint32_t*>(dst)[(int64_t)seq * inner + hj] = pack2(re * m, im * m);
    }
  } else {                                          // EPI_FRONT: gate and routing values
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int r = (is_mag ? tile - nq - na : tile - nq) * 16 + r0 + 8 * u;
      if (r < (is_mag ? p.rows_m : p.rows_a)) {
        const float bias = __bfloat162float(is_mag ? p.bias2[r] : p.bias[r]);
        p.gates[(int64_t)seq * (p.rows_a + p.rows_m) + (is_mag ? p.rows_a : 0) + r] = rbf((u ? sum.z : sum.x) + bias);
      }
    }
  }
}

// The tied head: 50 k real rows.  Every warp takes 16 rows over the whole of K (no reduction across warps); NT: groups of
// eight sequences.
template <int NT>
__global__ void __launch_bounds__(ST_THREADS, NT <= 2 ? 3 : 2) k_step_vocab(Skinny p) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ unsigned long long cand[ST_WARPS][NT * 8];
  __shared__ bool last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int xs_ld = row_ld(p.K >> 5);
  bf16* xs = reinterpret_cast<bf16*>(smem);
  pdl_trigger();
  const int tiles = (p.rows + 15) / 16, kb = p.K >> 5, r0 = lane >> 2, off = (lane & 3) * 8;
  const int stride = gridDim.x * ST_WARPS;
  int tile = warp * gridDim.x + blockIdx.x;         // neighbouring tiles on different SMs: the last wave is spread
  uint4 lo[ST_PF], hi[ST_PF];
  auto request = [&](int t) {
    const bf16 *wl = p.w + (int64_t)min(t * 16 + r0, p.rows - 1) * p.ld + off, *wh = p.w + (int64_t)min(t * 16 + r0 + 8, p.rows - 1) * p.ld + off;
#pragma unroll
    for (int i = 0; i < ST_PF; ++i)
      if (i < kb) {
        lo[i] = ld_weight(wl + i * 32);
        hi[i] = ld_weight(wh + i * 32);
      }
  };
  if (tile < tiles) request(tile);
  pdl_wait();
  load_rows<true>(p, xs, xs_ld, 0, p.K);
  __syncthreads();
  unsigned long long best[NT][2];
#pragma unroll
  for (int t = 0; t < NT; ++t) best[t][0] = best[t][1] = 0ull;
  for (; tile < tiles; tile += stride) {
    const bf16 *wl = p.w + (int64_t)min(tile * 16 + r0, p.rows - 1) * p.ld + off, *wh = p.w + (int64_t)min(tile * 16 + r0 + 8, p.rows - 1) * p.ld + off;
    float acc[NT][4];
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[t][j] = 0.f;
    for (int b = 0; b < kb; b += ST_PF) {
#pragma unroll
      for (int i = 0; i < ST_PF; ++i)
        if (b + i < kb) {
          block_mma<NT, false>(acc, lo[i], hi[i], xs, xs_ld, (b + i) * 32, lane);
          if (b + i + ST_PF < kb) {
            lo[i] = ld_weight(wl + (b + i + ST_PF) * 32);
            hi[i] = ld_weight(wh + (b + i + ST_PF) * 32);
          }
        }
    }
    if (tile + stride < tiles) request(tile + stride);
    const int ra = tile * 16 + r0, rb = ra + 8;
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int seq = t * 8 + (lane & 3) * 2 + c;
        if (p.logits) {
          if (seq < p.n) {
            if (ra < p.rows) p.logits[(int64_t)seq * p.ld_logits + ra] = __float2bfloat16_rn(acc[t][c]);
            if (rb < p.rows) p.logits[(int64_t)seq * p.ld_logits + rb] = __float2bfloat16_rn(acc[t][2 + c]);
          }
        } else {
          if (ra < p.rows) best[t][c] = max(best[t][c], best_key(acc[t][c], ra));
          if (rb < p.rows) best[t][c] = max(best[t][c], best_key(acc[t][2 + c], rb));
        }
      }
  }
  if (p.logits) return;
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      unsigned long long b = best[t][c];
      for (int o = 4; o < 32; o <<= 1) b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
      if (lane < 4) cand[warp][t * 8 + lane * 2 + c] = b;
    }
  __syncthreads();
  if (tid < p.n) {
    unsigned long long b = 0ull;
    for (int w = 0; w < ST_WARPS; ++w) b = max(b, cand[w][tid]);
    atomicMax(&p.best[tid], b);
    __threadfence();
  }
  __syncthreads();
  if (tid == 0) last = atomicAdd(p.done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (last && tid < p.n) {                          // the last CTA turns the maxima into token ids
    const unsigned long long b = *reinterpret_cast<volatile unsigned long long*>(&p.best[tid]);
    p.next_ids[tid] = (int64_t)(uint32_t)~(uint32_t)b;
  }
}

// Token embedding + embedding norm, one CTA per sequence; also clears the arg-max accumulators of this step.
__global__ void __launch_bounds__(1024) k_step_embed(const int64_t* __restrict__ ids, const bf16* __restrict__ er, const bf16* __restrict__ ei,
                                                     const float* __restrict__ scale, bf16* __restrict__ z, int D, int V,
                                                     unsigned long long* best, unsigned int* done) {
  __shared__ float s_part[32];
  pdl_trigger();
  pdl_wait();
  const int row = blockIdx.x, g = threadIdx.x, groups = D >> 2;
  const bool on = g < groups;
  if (g == 0) {
    best[row] = 0ull;
    if (row == 0) *done = 0u;
  }
  int64_t id = ids[row];
  id = id < 0 ? 0 : (id >= V ? V - 1 : id);
  float re[4] = {0.f, 0.f, 0.f, 0.f}, im[4] = {0.f, 0.f, 0.f, 0.f}, ss = 0.f;
  if (on) {
    E4<bf16>::ld(er + id * D + g * 4, re);
    E4<bf16>::ld(ei + id * D + g * 4, im);
#pragma unroll
    for (int j = 0; j < 4; ++j) ss += re[j] * re[j] + im[j] * im[j] + MAG_EPS;
  }
  ss = warp_sum(ss);
  if ((g & 31) == 0) s_part[g >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += s_part[w];
  if (!on) return;
  const float rrms = rsqrtf(tot / (float)D + 1e-6f);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const MagInv m_ = mag_inv(re[j] * re[j] + im[j] * im[j] + MAG_EPS);
    const float w = m_.mag * m_.inv * rrms * scale[g * 4 + j];
    re[j] *= w;
    im[j] *= w;
  }
  V4<bf16>::st(z + (int64_t)row * D * 2 + g * 8, re, im);
}

// Residual add + norm of a step with its own kernels, one CTA per sequence.
__global__ void __launch_bounds__(1024) k_step_norm(bf16* __restrict__ z, const bf16* __restrict__ delta, const float* __restrict__ res_scale,
                                                    const float* __restrict__ scale, bf16* __restrict__ xn, int D) {
  __shared__ float s_part[32];
  pdl_trigger();
  pdl_wait();
  const int64_t row = blockIdx.x;
  const int g = threadIdx.x, groups = D >> 2;
  const bool on = g < groups;
  float re[4] = {0.f, 0.f, 0.f, 0.f}, im[4] = {0.f, 0.f, 0.f, 0.f}, ss = 0.f;
  if (on) {
    V4<bf16>::ld(z + row * D * 2 + g * 8, re, im);
    if (delta) {
      const float s = *res_scale;
      float dr[4], di[4];
      V4<bf16>::ld(delta + row * D * 2 + g * 8, dr, di);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        re[j] = rbf(fmaf(s, dr[j], re[j]));
        im[j] = rbf(fmaf(s, di[j], im[j]));
      }
      V4<bf16>::st(z + row * D * 2 + g * 8, re, im);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) ss += re[j] * re[j] + im[j] * im[j] + MAG_EPS;
  }
  ss = warp_sum(ss);
  if ((g & 31) == 0) s_part[g >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += s_part[w];
  if (!on) return;
  const float rrms = rsqrtf(tot / (float)D + 1e-6f);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const MagInv m_ = mag_inv(re[j] * re[j] + im[j] * im[j] + MAG_EPS);
    const float w = m_.mag * m_.inv * rrms * scale[g * 4 + j];
    re[j] *= w;
    im[j] *= w;
  }
  V4<bf16>::st(xn + row * D * 2 + g * 8, re, im);
}

struct StepRecur {
  void* pool;
  const int32_t* slots;
  const bf16 *q, *k, *v;
  bf16* y;
  const float* gates;       // [n, G]
  const float *dt_bias, *dt_off;
  int64_t n_slots;
  int32_t L, layer, H, K, G, c_dt, c_pg, c_phase, c_score;
  float gamma_floor;
};

// The recurrent step on the slots (v11/model.py:927-965) with the gate arithmetic of v11/model.py:630-720 in front.  A CTA
// takes 16 of the 64 state rows of one (sequence, head), all K states at once: 16 bytes per thread and state, all in
// flight together.  (The pool-wide kernel gives a CTA all 64 rows; with a few sequences that leaves most SMs idle.)
template <typename S>
struct RecurRows {
  static constexpr int D = 64, NV = sizeof(S) == 2 ? 1 : 2;
  uint4 raw[QPAM_MAX_STATES][NV];
  float bias, decay[QPAM_MAX_STATES];
  S* base;                  // null: padded row of a captured batch

  // rows block * 16 .. + 15 of (seq, h); t: 0..255
  __device__ __forceinline__ void load(const StepRecur& p, int seq, int h, int block, int t) {
    const int slot = p.slots[seq];
    base = nullptr;
    if (slot < 0 || slot >= p.n_slots) return;
    base = reinterpret_cast<S*>(p.pool) + (((size_t)slot * p.L + p.layer) * p.K * p.H + h) * (size_t)(D * D * 2) +
           ((size_t)(block * 16 + (t >> 4)) * D + (t & 15) * 4) * 2;
    const size_t step = (size_t)p.H * D * D * 2;
#pragma unroll
    for (int k = 0; k < QPAM_MAX_STATES; ++k)
      if (k < p.K) {
#pragma unroll
        for (int i = 0; i < NV; ++i) raw[k][i] = __ldcs(reinterpret_cast<const uint4*>(base + k * step) + i);
        decay[k] = p.dt_off ? p.dt_off[k] : 0.f;
      }
    bias = p.dt_bias[h];
  }
  __device__ __forceinline__ void step(const StepRecur& p, int seq, int h, int block, int t) {
    const int row = block * 16 + (t >> 4), j0 = (t & 15) * 4;
    const size_t vb = ((size_t)seq * p.H + h) * D;
    if (!base) {            // no state, a defined output
      if ((t & 15) == 0) reinterpret_cast<uint32_t*>(p.y)[vb + row] = 0u;
      return;
    }
    const size_t step = (size_t)p.H * D * D * 2;
    float kr[4], ki[4], qr[4], qi[4];
    ldcg4(p.k + (vb + j0) * 2, kr, ki);
    ldcg4(p.q + (vb + j0) * 2, qr, qi);
    const float* g = p.gates + (int64_t)seq * p.G;
    float ph[QPAM_MAX_STATES], sc[QPAM_MAX_STATES];
    const float dt = __ldcg(g + p.c_dt + h) + bias, pg = p.c_pg >= 0 ? __ldcg(g + p.c_pg + h) : 0.f;
#pragma unroll
    for (int k = 0; k < QPAM_MAX_STATES; ++k) {
      ph[k] = p.c_phase >= 0 && k < p.K ? __ldcg(g + p.c_phase + h * p.K + k) : 0.f;
      sc[k] = p.c_score >= 0 && k < p.K ? __ldcg(g + p.c_score + h * p.K + k) : -INFINITY;
    }
    const uint32_t vw = __ldcg(reinterpret_cast<const uint32_t*>(p.v) + vb + row);
    const float prot = p.c_pg >= 0 ? sigmoidf_(pg) : 0.f, keep = 1.f - prot;
    const float2 v = make_float2(rbf(__uint_as_float(vw << 16) * keep), rbf(__uint_as_float(vw & 0xffff0000u) * keep));
    float wsum = 0.f;
    if (p.c_score >= 0) {
      const float wmax = fmaxf(fmaxf(sc[0], sc[1]), fmaxf(sc[2], sc[3]));
#pragma unroll
      for (int k = 0; k < QPAM_MAX_STATES; ++k) {
        sc[k] = __expf(sc[k] - wmax);
        wsum += sc[k];
      }
    }
    float yr = 0.f, yi = 0.f;
#pragma unroll
    for (int k = 0; k < QPAM_MAX_STATES; ++k) {
      if (k >= p.K) break;
      float gam = sigmoidf_(-(dt + decay[k]));        // exp(-softplus(x))
      if (p.gamma_floor > 0.f) gam = p.gamma_floor + (1.f - p.gamma_floor) * gam;
      gam = gam * (1.f - prot) + prot;
      float2 cf = make_float2(1.f, 0.f);
      if (p.c_phase >= 0) {
        const float w = p.c_score >= 0 ? sc[k] / wsum * (float)p.K : 1.f;
        float sn, cs;
        sincosf(ph[k], &sn, &cs);
        cf = make_float2(w * cs, w * sn);
      }
      float sr[4], si[4];
      S* cell = base + k * step;
      if constexpr (NV == 1) {
        const uint32_t w[4] = {raw[k][0].x, raw[k][0].y, raw[k][0].z, raw[k][0].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) { sr[j] = __uint_as_float(w[j] << 16); si[j] = __uint_as_float(w[j] & 0xffff0000u); }
      } else {
        const uint32_t w[8] = {raw[k][0].x, raw[k][0].y, raw[k][0].z, raw[k][0].w, raw[k][NV - 1].x, raw[k][NV - 1].y, raw[k][NV - 1].z, raw[k][NV - 1].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) { sr[j] = __uint_as_float(w[2 * j]); si[j] = __uint_as_float(w[2 * j + 1]); }
      }
      float pr = 0.f, pi = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        sr[j] = fmaf(gam, sr[j], v.x * kr[j] + v.y * ki[j]);                // v conj(k)
        si[j] = fmaf(gam, si[j], v.y * kr[j] - v.x * ki[j]);
        pr = fmaf(sr[j], qr[j], pr); pr = fmaf(-si[j], qi[j], pr);
        pi = fmaf(sr[j], qi[j], pi); pi = fmaf(si[j], qr[j], pi);
      }
      V4<S>::st(cell, sr, si);
      yr += cf.x * pr - cf.y * pi;
      yi += cf.x * pi + cf.y * pr;
    }
#pragma unroll
    for (int o = 8; o; o >>= 1) {
      yr += __shfl_xor_sync(0xffffffffu, yr, o);
      yi += __shfl_xor_sync(0xffffffffu, yi, o);
    }
    if ((t & 15) == 0) reinterpret_cast<uint32_t*>(p.y)[vb + row] = pack2(yr, yi);
}
};

template <typename S>
__global__ void __launch_bounds__(256) k_step_recur(StepRecur p) {
  pdl_trigger();
  pdl_wait();
  RecurRows<S> rr;
  rr.load(p, blockIdx.z, blockIdx.y, blockIdx.x, threadIdx.x);
  rr.step(p, blockIdx.z, blockIdx.y, blockIdx.x, threadIdx.x);
}

// ------------------------------------------------------------------------------------------------
// n <= 4: the whole step as ONE persistent kernel (a CTA per SM, cooperative launch), phases separated by grid barriers.
//
// At this size a kernel boundary (2.2 us from the last store to the first dependent load, measured in a graph with
// programmatic launch) costs as much as the work between two of them (1.5-2 us), and five boundaries per block were
// two thirds of the step.  A grid barrier is ~1 us, and the registers of a CTA carry over it: the weights of the next
// phase, and the recurrent states, are requested BEFORE the barrier, so HBM keeps streaming across it.  Every CTA keeps
// its own copy of the few rows of the residual stream in shared memory and forms residual add + norm redundantly.
// The wide projections are cut into units of 16 weight rows, one for each of a CTA's two groups of 8 warps; the projections
// back to D rows give a unit all 16 warps.  (Splitting their K over more CTAs, with fp32 partial sums added by every
// reader's prologue, cost more than it saved: 148 CTAs reading 36 KB each is 1 us of L2.)
// ------------------------------------------------------------------------------------------------
constexpr int ONE_THREADS = 512;
constexpr int QPAM_DEV_STEP_BARRIER = 241;

struct OneLayers {
  qpam_step_layer l[ST_ONE_LAYERS];
};
struct OneParams {
  const bf16 *embed_real, *embed_imag, *w_head, *b_head, *w_vocab;
  const float *embed_scale, *out_scale, *head_norm_scale, *rope;
  const int64_t *ids, *positions;
  const int32_t* slots;
  void* pool;
  int64_t* next_ids;
  bf16* logits;
  bf16 *gated, *q, *k, *v, *y;
  bf16 *delta, *head;           // [n, 2D]: the last block output, the head projection
  float* gates;
  unsigned long long* best;
  unsigned int *arrived, *done; // grid barrier, CTAs that have finished the head
  int64_t n_slots, rope_len, ld_logits;
  int32_t n, L, D, H, K, hidden, V, rows_a, rows_m;
  float q_scale;
};

struct OneUnit {
  const bf16 *wl, *wh;          // the lane's two weight rows
  int kb;                       // K blocks
};

// PAIR: at most two sequences, a unit of a projection back is 8 weight rows and their halves of K
template <typename S, bool PAIR>
struct One {
  const OneParams& p;
  const OneLayers& layers;
  // shared memory
  bf16 *z, *xs;                 // residual stream [4][2D] and normalised rows [4][xs_ld]
  bf16* xin;                    // input rows of a projection back to D rows; magnitudes
  float4* red;                  // [16][32]
  float* ssum;                  // [16]
  int xs_ld;
  // registers
  uint4 lo[ST_PF], hi[ST_PF];
  int tid, lane, warp, grp, gtid, gwarp, gidx, ngroups;
  unsigned int epoch;
  bool alive;

  __device__ __forceinline__ void group_sync() { asm volatile("bar.sync %0, 256;" ::"r"(grp + 1) : "memory"); }

  // All CTAs of the grid (cooperative launch: they are resident).  One counter and one polling thread per CTA: 1.2 us; a flag
  // per CTA, polled by 148 threads of each, took 8 us (22 k polls in flight delay the stores they wait for).  Bounded: a
  // barrier that is not reached within a second records a status and is not waited for again.
  // Arrival and wait are apart: what the next phase needs anyway is requested between them.
  __device__ __forceinline__ void grid_arrive() {
    __syncthreads();
    ++epoch;
    if (tid == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p.arrived) : "memory");
  }
  __device__ __forceinline__ void grid_wait() {
    bool ok = true;
    if (tid == 0 && alive) {
      const unsigned int target = epoch * gridDim.x;
      uint64_t t0 = 0;
      for (uint32_t it = 0;; ++it) {
        unsigned int v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p.arrived) : "memory");
        if (v >= target) break;
        if ((it & 255) == 255) {
          const uint64_t now = umma::global_ns();
          if (t0 == 0) t0 = now;
          else if (now - t0 > 1000000000ull) { ok = false; umma::record_device_error(QPAM_DEV_STEP_BARRIER); break; }
        }
      }
    }
    if (__syncthreads_or(!ok)) alive = false;
  }

  // weights of a unit from K block w on, for a warp that takes every nw-th
  __device__ __forceinline__ void request(const OneUnit& u, int w, int nw) {
    const int off = (lane & 3) * 8;
#pragma unroll
    for (int i = 0; i < ST_PF; ++i) {
      const int b = w + i * nw;
      if (b < u.kb) {
        lo[i] = ld_weight(u.wl + b * 32 + off);
        hi[i] = ld_weight(u.wh + b * 32 + off);
      }
    }
  }
  __device__ __forceinline__ void request(const OneUnit& u) { request(u, gwarp, ST_WARPS); }
  // acc += this warp's share (K blocks w, w + nw, ...) of one unit.  x holds the rows in shared memory.  SPLIT (n <= 2): the
  // unit is 8 weight rows, A rows 8..15 are their second half of K, whose inputs are columns 4..7.
  template <bool SPLIT>
  __device__ __forceinline__ void accumulate(const OneUnit& u, const bf16* x, int ld, int w, int nw, float (&acc)[4]) {
    float a[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};       // two chains of dependent MMAs
    const int col = lane >> 2;
    const bf16* xr = x + (SPLIT ? (size_t)((col >> 1) & 1) * ld + (col >> 2) * u.kb * 32 : (size_t)(col >> 1) * ld) + (lane & 3) * 8;
#pragma unroll 1
    for (int b = w;;) {
#pragma unroll
      for (int i = 0; i < ST_PF; ++i) {
        const int bi = b + i * nw;
        if (bi < u.kb) {
          uint4 v = *reinterpret_cast<const uint4*>(xr + bi * 32);
          if (col & 1) { v.x = rot(v.x); v.y = rot(v.y); v.z = rot(v.z); v.w = rot(v.w); }
          mma16816(a[0], lo[i].x, hi[i].x, lo[i].y, hi[i].y, v.x, v.y);
          mma16816(a[1], lo[i].z, hi[i].z, lo[i].w, hi[i].w, v.z, v.w);
        }
      }
      b += ST_PF * nw;
      if (b >= u.kb) break;
      request(u, b, nw);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[j] = a[0][j] + a[1][j];
  }
  // A unit of this group of 8 warps; sums valid in the group's first warp: (x, y) = (re, im) of row lane / 4, (z, w) of row
  // lane / 4 + 8, for sequence lane & 3.
  __device__ __forceinline__ float4 group_product(const OneUnit& u, const bf16* x, int ld) {
    float acc[4];
    accumulate<false>(u, x, ld, gwarp, ST_WARPS, acc);
    group_sync();                       // the previous unit's sums have been read
    red[warp * 32 + lane] = make_float4(acc[0], acc[1], acc[2], acc[3]);
    group_sync();
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    if (gwarp == 0) {
#pragma unroll
      for (int w = 0; w < ST_WARPS; ++w) {
        const float4 o = red[(grp * ST_WARPS + w) * 32 + lane];
        s.x += o.x; s.y += o.y; s.z += o.z; s.w += o.w;
      }
    }
    return s;
  }

  // ---- units of the phases
  __device__ __forceinline__ OneUnit unit_gu(int l, int u) const {
    const bf16* w = (const bf16*)layers.l[l].w_gu;
    const int64_t ld = 2 * p.D;
    const int r = u * 8 + (lane >> 2);
    return {w + 2 * (int64_t)r * ld, w + 2 * (int64_t)(p.hidden + r) * ld, p.D >> 4};
  }
  __device__ __forceinline__ OneUnit unit_back(const void* w_, int kblocks, int u) const {    // a projection back to D rows
    const int64_t ld = (int64_t)kblocks * 32;
    if (PAIR) {
      const bf16* w = (const bf16*)w_ + 2 * (int64_t)(u * 8 + (lane >> 2)) * ld;
      return {w, w + (ld >> 1), kblocks >> 1};
    }
    const bf16* w = (const bf16*)w_ + 2 * (int64_t)(u * 16 + (lane >> 2)) * ld;
    return {w, w + 16 * ld, kblocks};
  }
  __device__ __forceinline__ int units_back() const { return PAIR ? p.D / 8 : p.D / 16; }
  __device__ __forceinline__ void request_back(const void* w, int kblocks) {
    if ((int)blockIdx.x < units_back()) request(unit_back(w, kblocks, blockIdx.x), warp, 16);
  }
  __device__ __forceinline__ OneUnit unit_front(int l, int u) const {
    const qpam_step_layer& y = layers.l[l];
    const int nq = 3 * p.H * 4, na = (p.rows_a + 15) / 16, r0 = lane >> 2;
    const int64_t ld = 2 * p.D;
    const bf16* w = (const bf16*)y.w_front;
    if (u < nq) {
      w += 2 * (int64_t)(u * 16 + r0) * ld;
      return {w, w + 16 * ld, p.D >> 4};
    }
    if (u < nq + na) {
      const int t = (u - nq) * 16;
      w += (int64_t)6 * p.H * 64 * ld;
      return {w + min(t + r0, p.rows_a - 1) * ld, w + min(t + r0 + 8, p.rows_a - 1) * ld, p.D >> 4};
    }
    const int t = (u - nq - na) * 16;
    const bf16* wm = (const bf16*)y.w_mag;
    return {wm + (int64_t)min(t + r0, p.rows_m - 1) * p.D, wm + (int64_t)min(t + r0 + 8, p.rows_m - 1) * p.D, p.D >> 5};
  }
  __device__ __forceinline__ int units_front() const { return 3 * p.H * 4 + (p.rows_a + 15) / 16 + (p.rows_m + 15) / 16; }

  // ---- residual add + norm of the few rows, by the whole CTA: a row gets 16 / (1, 2, 4) warps, a thread two complex
  // values at a time.  DELTA: z += scale * delta; otherwise z stands.  HEAD: z is replaced by delta, and the normalised row
  // goes out as [re | im] planes.
  template <bool DELTA, bool HEAD>
  __device__ __forceinline__ void norm_rows(const bf16* delta, const float* scale_ptr, const float* norm_scale) {
    const int wpr = p.n == 1 ? 16 : p.n == 2 ? 8 : 4;
    const int r = warp / wpr, t = (warp - r * wpr) * 32 + lane, nt = wpr * 32;
    const int pairs = r < p.n ? p.D >> 1 : 0;
    float ss = 0.f;
    const float s = DELTA && !HEAD ? __ldg(scale_ptr) : 1.f;
#pragma unroll 1
    for (int g = t; g < pairs; g += nt) {
      uint2 d = make_uint2(0u, 0u);
      if (DELTA) d = __ldcg(reinterpret_cast<const uint2*>(delta + (size_t)r * 2 * p.D + g * 4));
      uint2* zp = reinterpret_cast<uint2*>(z + (size_t)r * 2 * p.D + g * 4);
      uint2 w = HEAD ? d : *zp;
      if (DELTA && !HEAD) {
        w = make_uint2(pack2(fmaf(s, __uint_as_float(d.x << 16), __uint_as_float(w.x << 16)), fmaf(s, __uint_as_float(d.x & 0xffff0000u), __uint_as_float(w.x & 0xffff0000u))),
                       pack2(fmaf(s, __uint_as_float(d.y << 16), __uint_as_float(w.y << 16)), fmaf(s, __uint_as_float(d.y & 0xffff0000u), __uint_as_float(w.y & 0xffff0000u))));
      }
      if (DELTA) *zp = w;
      const float v0 = __uint_as_float(w.x << 16), v1 = __uint_as_float(w.x & 0xffff0000u), v2 = __uint_as_float(w.y << 16), v3 = __uint_as_float(w.y & 0xffff0000u);
      ss += v0 * v0 + v1 * v1 + v2 * v2 + v3 * v3 + 2.f * MAG_EPS;
    }
    finish_norm<HEAD>(ss, r, t, nt, wpr, pairs, norm_scale, xs, xs_ld);
  }
  // norm of z (whose squares this thread has summed) into rows of `ld` scalars
  template <bool PLANAR>
  __device__ __forceinline__ void finish_norm(float ss, int r, int t, int nt, int wpr, int pairs, const float* norm_scale, bf16* dst, int ld) {
    float2 sc = make_float2(0.f, 0.f);
    if (t < pairs) sc = *reinterpret_cast<const float2*>(norm_scale + t * 2);
    ss = warp_sum(ss);
    if (lane == 0) ssum[warp] = ss;
    __syncthreads();
    float tot = ssum[(r * wpr + (lane & (wpr - 1))) & 15];
    for (int o = wpr >> 1; o; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
    const float rrms = rsqrtf(tot / (float)p.D + 1e-6f);
#pragma unroll 1
    for (int g = t; g < pairs; g += nt) {
      if (g != t) sc = *reinterpret_cast<const float2*>(norm_scale + g * 2);
      const uint2 w = *reinterpret_cast<const uint2*>(z + (size_t)r * 2 * p.D + g * 4);
      const float a = __uint_as_float(w.x << 16), b = __uint_as_float(w.x & 0xffff0000u), c = __uint_as_float(w.y << 16), d = __uint_as_float(w.y & 0xffff0000u);
      const MagInv m0 = mag_inv(a * a + b * b + MAG_EPS), m1 = mag_inv(c * c + d * d + MAG_EPS);
      const float w0 = m0.mag * m0.inv * rrms * sc.x, w1 = m1.mag * m1.inv * rrms * sc.y;
      if (PLANAR) {
        *reinterpret_cast<uint32_t*>(dst + (size_t)r * ld + g * 2) = pack2(a * w0, c * w1);
        *reinterpret_cast<uint32_t*>(dst + (size_t)r * ld + p.D + g * 2) = pack2(b * w0, d * w1);
      } else {
        *reinterpret_cast<uint2*>(dst + (size_t)r * ld + g * 4) = make_uint2(pack2(a * w0, b * w0), pack2(c * w1, d * w1));
      }
    }
    __syncthreads();
  }

  // ---- token embedding + its norm: the residual stream of this CTA
  __device__ __forceinline__ void embed() {
    const int wpr = p.n == 1 ? 16 : p.n == 2 ? 8 : 4;
    const int r = warp / wpr, t = (warp - r * wpr) * 32 + lane, nt = wpr * 32;
    const int pairs = r < p.n ? p.D >> 1 : 0;
    int64_t id = pairs ? p.ids[r] : 0;
    id = id < 0 ? 0 : (id >= p.V ? p.V - 1 : id);
    float ss = 0.f;
#pragma unroll 1
    for (int g = t; g < pairs; g += nt) {
      const uint32_t a = *reinterpret_cast<const uint32_t*>(p.embed_real + id * p.D + g * 2), b = *reinterpret_cast<const uint32_t*>(p.embed_imag + id * p.D + g * 2);
      *reinterpret_cast<uint2*>(z + (size_t)r * 2 * p.D + g * 4) = make_uint2(__byte_perm(a, b, 0x5410), __byte_perm(a, b, 0x7632));
      const float v0 = __uint_as_float(a << 16), v1 = __uint_as_float(b << 16), v2 = __uint_as_float(a & 0xffff0000u), v3 = __uint_as_float(b & 0xffff0000u);
      ss += v0 * v0 + v1 * v1 + v2 * v2 + v3 * v3 + 2.f * MAG_EPS;
    }
    finish_norm<false>(ss, r, t, nt, wpr, pairs, p.embed_scale, z, 2 * p.D);
  }

  // ---- a projection back to D complex rows, all 16 warps on a unit whose first weights have been requested.  x: [n, 32 *
  // kblocks] in global memory (written by other CTAs), or null for the normalised rows this CTA holds.
  __device__ __forceinline__ void project_back(const void* w, int kblocks, const bf16* x, const bf16* bias, bf16* out) {
    if ((int)blockIdx.x >= units_back()) return;
    const int ld = x ? row_ld(kblocks) : xs_ld;
    if (x) {
      const int vec = kblocks * 4;
      for (int i = tid; i < p.n * vec; i += ONE_THREADS) {
        const int r = i / vec, g = i - r * vec;
        *reinterpret_cast<uint4*>(xin + (size_t)r * ld + g * 8) = __ldcg(reinterpret_cast<const uint4*>(x + (size_t)r * kblocks * 32 + g * 8));
      }
      __syncthreads();
    }
    const bf16* rows = x ? xin : xs;
    for (int u = blockIdx.x; u < units_back(); u += gridDim.x) {
      const OneUnit un = unit_back(w, kblocks, u);
      if (u != (int)blockIdx.x) request(un, warp, 16);
      float acc[4];
      accumulate<PAIR>(un, rows, ld, warp, 16, acc);
      __syncthreads();
      red[warp * 32 + lane] = make_float4(acc[0], acc[1], acc[2], acc[3]);
      __syncthreads();
      if (warp == 0) {
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float4 o = red[i * 32 + lane];
          s.x += o.x; s.y += o.y; s.z += o.z; s.w += o.w;
        }
        const int seq = lane & 3;
        uint32_t* o = reinterpret_cast<uint32_t*>(out);
        if (PAIR) {                     // (x, y) of columns 0..3 and (z, w) of columns 4..7 are the halves of K
          const float re = s.x + __shfl_xor_sync(0xffffffffu, s.z, 2), im = s.y + __shfl_xor_sync(0xffffffffu, s.w, 2);
          const int row = u * 8 + (lane >> 2);
          if (seq < p.n) store_row(o, seq, row, re, im, bias);
        } else if (seq < p.n) {
          const int row = u * 16 + (lane >> 2);
          store_row(o, seq, row, s.x, s.y, bias);
          store_row(o, seq, row + 8, s.z, s.w, bias);
        }
      }
    }
  }
  __device__ __forceinline__ void store_row(uint32_t* out, int seq, int row, float re, float im, const bf16* bias) {
    if (bias) {
      const uint32_t b = reinterpret_cast<const uint32_t*>(bias)[row];
      re += __uint_as_float(b << 16);
      im += __uint_as_float(b & 0xffff0000u);
    }
    out[(size_t)seq * p.D + row] = pack2(re, im);
  }
};

template <typename S, bool PAIR>
__global__ void __launch_bounds__(ONE_THREADS, 1) k_step_one(const __grid_constant__ OneParams p, const __grid_constant__ OneLayers layers) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ float ssum[16];
  __shared__ bool last_s;
  __shared__ unsigned long long cand[16][4];
  One<S, PAIR> m{p, layers};
  const int tid = threadIdx.x, lane = tid & 31;
  m.tid = tid; m.lane = lane; m.warp = tid >> 5; m.grp = tid >> 8; m.gtid = tid & 255; m.gwarp = m.gtid >> 5;
  m.gidx = m.grp * gridDim.x + blockIdx.x; m.ngroups = 2 * gridDim.x;
  m.epoch = 0; m.alive = true; m.ssum = ssum;
  const int kb_down = p.hidden >> 4, kb_o = p.H * 4, kb_D = p.D >> 4;
  m.xs_ld = row_ld(kb_D);
  m.z = reinterpret_cast<bf16*>(smem);
  m.xs = m.z + (size_t)4 * 2 * p.D;
  m.red = reinterpret_cast<float4*>(m.xs + (size_t)4 * m.xs_ld);
  m.xin = reinterpret_cast<bf16*>(m.red + 16 * 32);
  const int n = p.n, inner = p.H * 64;
  const int seq = lane & 3, r0 = lane >> 2;      // what this lane holds of a unit's sums
  const bool first_warp = m.gwarp == 0;

  if (m.gidx < p.hidden / 8) m.request(m.unit_gu(0, m.gidx));
  m.embed();
  m.template norm_rows<false, false>(nullptr, nullptr, layers.l[0].n1);
  // Half a layer at a time (gated unit, sequence mixing): both are a norm, a wide projection and one back to D rows.  One copy of
  // that code serves both and stays in the instruction cache; written out per layer it missed 620 times a layer, now 385 (a step of one sequence 279 -> 267 us).
#pragma unroll 1
  for (int half = 0; half < 2 * p.L; ++half) {
    const int l = half >> 1;
    const bool mixing = half & 1;
    const qpam_step_layer& y = layers.l[l];
    if (half > 0) m.template norm_rows<true, false>(p.delta, mixing ? y.cgu_scale : layers.l[l - 1].pam_scale, mixing ? y.n2 : y.n1);
    if (!mixing) {
      // ---- gate | up projections and the gated unit
      for (int u = m.gidx; u < p.hidden / 8; u += m.ngroups) {
        const OneUnit un = m.unit_gu(l, u);
        if (u != m.gidx) m.request(un);
        const int ch = u * 8 + r0;
        const float bias = y.act_bias[ch], beta = y.act_beta ? y.act_beta[ch] : 0.f;
        const float4 s = m.group_product(un, m.xs, m.xs_ld);
        if (first_warp && seq < n) {
          const float gr = rbf(s.x), gi = rbf(s.y), ur = rbf(s.z), ui = rbf(s.w);
          const MagInv um = mag_inv(ur * ur + ui * ui + MAG_EPS), gm = mag_inv(gr * gr + gi * gi + MAG_EPS);
          const float act = y.act_beta ? um.mag * sigmoidf_(beta * um.mag + bias) : fmaxf(um.mag + bias, 0.f);
          const float h = sigmoidf_(gm.mag) * gm.inv * act * um.inv;
          reinterpret_cast<uint32_t*>(p.gated)[(int64_t)seq * p.hidden + ch] = pack2((gr * ur - gi * ui) * h, (gr * ui + gi * ur) * h);
        }
      }
    } else {
      // ---- q, k, v and the gate values
      const int nq = 3 * p.H * 4, na = (p.rows_a + 15) / 16;
      for (int u = m.gidx; u < m.units_front(); u += m.ngroups) {
        const OneUnit un = m.unit_front(l, u);
        if (u != m.gidx) m.request(un);
        const bool mag = u >= nq + na;
        const bf16* x = m.xs;
        int ld = m.xs_ld;
        float2 rc[2] = {make_float2(1.f, 0.f), make_float2(1.f, 0.f)};
        if (u < 2 * p.H * 4 && p.rope && seq < n) {
          int64_t pos = p.positions[seq];
          pos = pos < 0 ? 0 : (pos >= p.rope_len ? p.rope_len - 1 : pos);
          const float2* rp = reinterpret_cast<const float2*>(p.rope) + pos * 64 + (u * 16 + r0) % 64;
          rc[0] = rp[0];
          rc[1] = rp[8];
        }
        if (mag) {                              // rows that read |xn|: magnitudes of the rounded rows, in the group's own slice
          ld = row_ld(p.D >> 5);
          bf16* mg = m.xin + (size_t)m.grp * 4 * ld;
          for (int i = m.gtid; i < n * (p.D >> 1); i += 256) {
            const int r = i / (p.D >> 1), g = i - r * (p.D >> 1);
            const uint2 w = *reinterpret_cast<const uint2*>(m.xs + (size_t)r * m.xs_ld + g * 4);
            const float a = __uint_as_float(w.x << 16), b = __uint_as_float(w.x & 0xffff0000u), c = __uint_as_float(w.y << 16), d = __uint_as_float(w.y & 0xffff0000u);
            *reinterpret_cast<uint32_t*>(mg + (size_t)r * ld + g * 2) = pack2(fsqrt_(a * a + b * b + MAG_EPS), fsqrt_(c * c + d * d + MAG_EPS));
          }
          m.group_sync();
          x = mg;
        }
        const float4 s = m.group_product(un, x, ld);
        if (first_warp && seq < n) {
          if (u < nq) {
            const int which = u / (p.H * 4), hj = u * 16 + r0 - which * inner;
            const float mul = which == 0 ? p.q_scale : 1.f;
            uint32_t* dst = reinterpret_cast<uint32_t*>(which == 0 ? p.q : which == 1 ? p.k : p.v) + (int64_t)seq * inner + hj;
            dst[0] = pack2((s.x * rc[0].x - s.y * rc[0].y) * mul, (s.x * rc[0].y + s.y * rc[0].x) * mul);
            dst[8] = pack2((s.z * rc[1].x - s.w * rc[1].y) * mul, (s.z * rc[1].y + s.w * rc[1].x) * mul);
          } else {
            const int rows = mag ? p.rows_m : p.rows_a, r = (mag ? u - nq - na : u - nq) * 16 + r0;
            const bf16* bb = mag ? (const bf16*)y.b_mag : (const bf16*)y.b_front + 6 * inner;
            float* o = p.gates + (int64_t)seq * (p.rows_a + p.rows_m) + (mag ? p.rows_a : 0);
            if (r < rows) o[r] = rbf(s.x + __bfloat162float(bb[r]));
            if (r + 8 < rows) o[r + 8] = rbf(s.z + __bfloat162float(bb[r + 8]));
          }
        }
      }
      // ---- recurrent step: a unit is 16 state rows of one (sequence, head), all K states
      StepRecur sr;
      sr.pool = p.pool; sr.slots = p.slots; sr.q = p.q; sr.k = p.k; sr.v = p.v; sr.y = p.y; sr.gates = p.gates; sr.dt_bias = y.dt_bias; sr.dt_off = y.dt_off;
      sr.n_slots = p.n_slots; sr.L = p.L; sr.layer = l; sr.H = p.H; sr.K = p.K; sr.G = p.rows_a + p.rows_m; sr.c_dt = y.col_dt; sr.c_pg = y.col_pg;
      sr.c_phase = p.K > 1 ? y.col_phase : -1; sr.c_score = y.col_score; sr.gamma_floor = y.gamma_floor;
      m.grid_arrive();
      RecurRows<S> rr;
      const int recur_units = n * p.H * 4;
      if (m.gidx < recur_units) rr.load(sr, m.gidx / (4 * p.H), (m.gidx >> 2) % p.H, m.gidx & 3, m.gtid);
      m.grid_wait();
#pragma unroll 1
      for (int u = m.gidx; u < recur_units; u += m.ngroups) {
        if (u != m.gidx) rr.load(sr, u / (4 * p.H), (u >> 2) % p.H, u & 3, m.gtid);
        rr.step(sr, u / (4 * p.H), (u >> 2) % p.H, u & 3, m.gtid);
      }
    }
    // ---- down or output projection
    const void* w = mixing ? y.w_o : y.w_down;
    const int kb = mixing ? kb_o : kb_down;
    m.grid_arrive();
    m.request_back(w, kb);
    m.grid_wait();
    m.project_back(w, kb, mixing ? p.y : p.gated, nullptr, p.delta);
    m.grid_arrive();
    if (half + 1 == 2 * p.L) m.request_back(p.w_head, kb_D);
    else if (m.gidx < (mixing ? p.hidden / 8 : m.units_front())) m.request(mixing ? m.unit_gu(l + 1, m.gidx) : m.unit_front(l, m.gidx));
    m.grid_wait();
  }
  // ---- head projection (its output has a buffer of its own: slower CTAs still read the last block's)
  m.template norm_rows<true, false>(p.delta, layers.l[p.L - 1].pam_scale, p.out_scale);
  m.project_back(p.w_head, kb_D, nullptr, p.b_head, p.head);
  // ---- tied head: a warp takes 16 vocabulary rows over all of K
  const int tiles = (p.V + 15) / 16, stride = gridDim.x * 16, off = (lane & 3) * 8;
  int tile = m.warp * gridDim.x + blockIdx.x;
  auto row_ptr = [&](int t, int h) { return p.w_vocab + (int64_t)min(t * 16 + r0 + h, p.V - 1) * 2 * p.D + off; };
  auto request = [&](int t) {
#pragma unroll
    for (int i = 0; i < ST_PF; ++i)
      if (i < kb_D) {
        m.lo[i] = ld_weight(row_ptr(t, 0) + i * 32);
        m.hi[i] = ld_weight(row_ptr(t, 8) + i * 32);
      }
  };
  m.grid_arrive();
  if (tile < tiles) request(tile);
  m.grid_wait();
  m.template norm_rows<true, true>(p.head, nullptr, p.head_norm_scale);
  unsigned long long best[2] = {0ull, 0ull};
  for (; tile < tiles; tile += stride) {
    const bf16 *wl = row_ptr(tile, 0), *wh = row_ptr(tile, 8);
    float acc[1][4] = {{0.f, 0.f, 0.f, 0.f}};
    for (int b = 0; b < kb_D; b += ST_PF) {
#pragma unroll
      for (int i = 0; i < ST_PF; ++i)
        if (b + i < kb_D) {
          block_mma<1, false>(acc, m.lo[i], m.hi[i], m.xs, m.xs_ld, (b + i) * 32, lane);
          if (b + i + ST_PF < kb_D) {
            m.lo[i] = ld_weight(wl + (b + i + ST_PF) * 32);
            m.hi[i] = ld_weight(wh + (b + i + ST_PF) * 32);
          }
        }
    }
    if (tile + stride < tiles) request(tile + stride);
    const int ra = tile * 16 + r0, rb = ra + 8;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int sq = (lane & 3) * 2 + c;
      if (p.logits) {
        if (sq < n) {
          if (ra < p.V) p.logits[(int64_t)sq * p.ld_logits + ra] = __float2bfloat16_rn(acc[0][c]);
          if (rb < p.V) p.logits[(int64_t)sq * p.ld_logits + rb] = __float2bfloat16_rn(acc[0][2 + c]);
        }
      } else {
        if (ra < p.V) best[c] = max(best[c], best_key(acc[0][c], ra));
        if (rb < p.V) best[c] = max(best[c], best_key(acc[0][2 + c], rb));
      }
    }
  }
  if (p.logits) return;
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    unsigned long long b = best[c];
    for (int o = 4; o < 32; o <<= 1) b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
    if (lane < 2) cand[m.warp][lane * 2 + c] = b;
  }
  __syncthreads();
  if (tid < n) {
    unsigned long long b = 0ull;
    for (int w = 0; w < 16; ++w) b = max(b, cand[w][tid]);
    atomicMax(&p.best[tid], b);
    __threadfence();
  }
  __syncthreads();
  if (tid == 0) last_s = atomicAdd(p.done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (last_s && tid < n) {
    __threadfence();
    p.next_ids[tid] = (int64_t)(uint32_t)~(uint32_t)*reinterpret_cast<volatile unsigned long long*>(&p.best[tid]);
  }
}

// ------------------------------------------------------------------------------------------------ host
template <typename... Params, typename... Args>
int launch_pdl(const char* name, void (*kern)(Params...), dim3 grid, int threads, size_t smem, int cluster, cudaStream_t st, Args... args) {
  const int rc = allow_smem(reinterpret_cast<const void*>(kern), smem);
  if (rc) return rc;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = cluster;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, args...);
  if (e != cudaSuccess) return cuda_fail(e, name);
  note_launch(name, st);
  return QPAM_OK;
}

// Cluster size that splits K so that a projection with few rows still covers the SMs
int split_of(int tiles, int kblocks) {
  int cs = 1;
  while (cs < 8 && tiles * cs < sm_count() && kblocks / (cs * 2) >= ST_WARPS / 2) cs *= 2;
  return cs;
}

template <int EPI>
int launch_proj(const Skinny& p, int tiles, cudaStream_t st) {
  const int nt = p.n <= 4 ? 1 : p.n <= 8 ? 2 : 4;
  const int cs = EPI == EPI_COMPLEX ? split_of(tiles, p.K / 32) : 1;
  const int kb = (p.K / 32 + cs - 1) / cs;
  const size_t smem = (size_t)nt * 4 * row_ld(kb) * sizeof(bf16) + (size_t)ST_WARPS * nt * 32 * sizeof(float4);
  const dim3 grid(tiles * cs);
  if (nt == 1) return launch_pdl("k_step_proj", k_step_proj<1, EPI>, grid, ST_THREADS, smem, cs, st, p);
  if (nt == 2) return launch_pdl("k_step_proj", k_step_proj<2, EPI>, grid, ST_THREADS, smem, cs, st, p);
  return launch_pdl("k_step_proj", k_step_proj<4, EPI>, grid, ST_THREADS, smem, cs, st, p);
}

int launch_vocab(const Skinny& p, cudaStream_t st) {
  const int nt = p.n <= 8 ? 1 : 2;
  const size_t smem = (size_t)nt * 8 * row_ld(p.K / 32) * sizeof(bf16);
  const int per_sm = smem * 3 <= 200 * 1024 ? (nt <= 2 ? 3 : 2) : smem * 2 <= 200 * 1024 ? 2 : 1;
  const int tiles = (p.rows + 15) / 16;
  const dim3 grid(min(sm_count() * per_sm, (tiles + ST_WARPS - 1) / ST_WARPS));
  if (nt == 1) return launch_pdl("k_step_vocab", k_step_vocab<1>, grid, ST_THREADS, smem, 1, st, p);
  return launch_pdl("k_step_vocab", k_step_vocab<2>, grid, ST_THREADS, smem, 1, st, p);
}

struct StepWs;
int launch_one(const qpam_step_args* a, const StepWs& w, cudaStream_t st);

struct StepWs {
  bf16 *z, *gated, *delta, *xn, *q, *k, *v, *y;
  float* gates;
  unsigned long long* best;
  unsigned int* done;         // done[0]: CTAs that have finished the head, done[32]: grid barrier
  size_t bytes;
};
StepWs carve(const qpam_step_args* a, void* base) {
  StepWs w;
  size_t at = 0;
  auto take = [&](size_t bytes) { void* r = (char*)base + at; at += (bytes + 255) & ~(size_t)255; return r; };
  const size_t n = a->n, D2 = 2 * (size_t)a->D, I2 = 2 * (size_t)a->H * 64;
  w.z = (bf16*)take(n * D2 * 2);
  w.delta = (bf16*)take(n * D2 * 2);
  w.xn = (bf16*)take(n * D2 * 2);
  w.gated = (bf16*)take(n * 2 * (size_t)a->hidden * 2);
  w.q = (bf16*)take(n * I2 * 2);
  w.k = (bf16*)take(n * I2 * 2);
  w.v = (bf16*)take(n * I2 * 2);
  w.y = (bf16*)take(n * I2 * 2);
  w.gates = (float*)take(n * (size_t)(a->rows_a + a->rows_m) * 4);
  w.best = (unsigned long long*)take(n * 8 + 256);   // (one piece with the counters: cleared together)
  w.done = (unsigned int*)(w.best + n);
  w.bytes = at;
  return w;
}

int launch_one(const qpam_step_args* a, const StepWs& w, cudaStream_t st) {
  OneParams p{};
  p.embed_real = (const bf16*)a->embed_real; p.embed_imag = (const bf16*)a->embed_imag; p.w_head = (const bf16*)a->w_head; p.b_head = (const bf16*)a->b_head;
  p.w_vocab = (const bf16*)a->w_vocab; p.embed_scale = a->embed_scale; p.out_scale = a->out_scale; p.head_norm_scale = a->head_norm_scale; p.rope = a->rope;
  p.ids = a->ids; p.positions = a->positions; p.slots = a->slot_ids; p.pool = a->pool; p.next_ids = a->next_ids; p.logits = (bf16*)a->logits;
  p.gated = w.gated; p.q = w.q; p.k = w.k; p.v = w.v; p.y = w.y; p.gates = w.gates; p.delta = w.delta; p.head = w.xn; p.best = w.best; p.done = w.done; p.arrived = w.done + 32;
  p.n_slots = a->n_slots; p.rope_len = a->rope_len; p.ld_logits = a->ld_logits; p.n = a->n; p.L = a->n_layers; p.D = a->D; p.H = a->H; p.K = a->K;
  p.hidden = a->hidden; p.V = a->V; p.rows_a = a->rows_a; p.rows_m = a->rows_m; p.q_scale = a->q_scale;
  const int grid = sm_count();
  OneLayers layers{};
  for (int l = 0; l < a->n_layers; ++l) layers.l[l] = a->layers[l];
  const size_t rows_in = (size_t)4 * max(row_ld(max(a->hidden >> 4, a->H * 4)), 2 * row_ld(a->D >> 5));   // block inputs, or magnitudes of both groups
  const size_t smem = ((size_t)4 * 2 * a->D + 4 * row_ld(a->D >> 4) + rows_in) * sizeof(bf16) + (size_t)16 * 32 * sizeof(float4);
  QPAM_CUDA(cudaMemsetAsync(w.best, 0, (size_t)a->n * 8 + 256, st));
  void* args[] = {&p, &layers};
  const bool pair = a->n <= 2;
  auto kern = a->state_dtype == QPAM_F32 ? pair ? (const void*)k_step_one<float, true> : (const void*)k_step_one<float, false>
                                         : pair ? (const void*)k_step_one<bf16, true> : (const void*)k_step_one<bf16, false>;
  const int rc = allow_smem(kern, smem);
  if (rc) return rc;
  QPAM_CUDA(cudaLaunchCooperativeKernel(kern, dim3(grid), dim3(ONE_THREADS), args, smem, st));
  QPAM_LAUNCH_CHECK("k_step_one");
  return QPAM_OK;
}

}  // namespace
}  // namespace qpam

using namespace qpam;

namespace qpam {
int step_device_status(int* value, bool clear) {
  QPAM_CUDA(umma::read_device_error(value, clear));
  return QPAM_OK;
}
}  // namespace qpam

extern "C" int32_t qpam_step_supported(int32_t n, int32_t D, int32_t H, int32_t d, int32_t K, int32_t hidden, int32_t V) {
  return n >= 1 && n <= 16 && D >= 32 && D % 32 == 0 && D <= 1024 && d == 64 && H >= 1 && H <= 64 && K >= 1 && K <= QPAM_MAX_STATES && hidden % 32 == 0 &&
         hidden >= 32 && hidden <= 8192 && V >= 1;
}

extern "C" size_t qpam_step_workspace_bytes(const qpam_step_args* a) { return a ? carve(a, nullptr).bytes : 0; }

extern "C" int qpam_step_fwd(const qpam_step_args* a, void* stream) {
  QPAM_REQUIRE(a, "step: NULL args");
  QPAM_REQUIRE(qpam_step_supported(a->n, a->D, a->H, a->d, a->K, a->hidden, a->V), "step: shape not covered (n=%d D=%d H=%d d=%d K=%d hidden=%d)",
               a->n, a->D, a->H, a->d, a->K, a->hidden);
  QPAM_REQUIRE(a->layers && a->n_layers >= 1 && a->embed_real && a->embed_imag && a->embed_scale && a->out_scale && a->head_norm_scale && a->w_head &&
                   a->w_vocab && a->ids && a->slot_ids && a->pool, "step: NULL pointer argument");
  QPAM_REQUIRE(!a->rope || (a->positions && a->rope_len > 0), "step: the rotary table needs positions");
  QPAM_REQUIRE((a->next_ids != nullptr) != (a->logits != nullptr), "step: exactly one of next_ids and logits");
  QPAM_REQUIRE(!a->logits || a->ld_logits >= a->V, "step: logits rows are too short");
  QPAM_REQUIRE(a->state_dtype == QPAM_F32 || a->state_dtype == QPAM_BF16, "step: state_dtype %d unknown", a->state_dtype);
  QPAM_REQUIRE(a->rows_a >= a->H && a->rows_m >= 0, "step: bad gate rows");
  QPAM_REQUIRE(a->workspace && a->workspace_bytes >= qpam_step_workspace_bytes(a), "step: workspace too small");
  for (int l = 0; l < a->n_layers; ++l) {
    const qpam_step_layer& y = a->layers[l];
    QPAM_REQUIRE(y.w_gu && y.w_down && y.w_front && y.b_front && y.w_o && y.n1 && y.n2 && y.act_bias && y.cgu_scale && y.pam_scale && y.dt_bias,
                 "step: NULL pointer in layer %d", l);
    QPAM_REQUIRE((a->rows_m == 0 || (y.w_mag && y.b_mag)) && y.col_dt >= 0, "step: missing gate weights in layer %d", l);
    QPAM_REQUIRE(a->K == 1 || (y.col_phase >= 0 && y.dt_off), "step: K > 1 needs phases and decay offsets");
  }
  cudaStream_t st = (cudaStream_t)stream;
  const StepWs w = carve(a, a->workspace);
  if (a->n <= ST_ONE_N && a->n_layers <= ST_ONE_LAYERS) return launch_one(a, w, st);
  const int n = a->n, D = a->D, H = a->H, K2 = 2 * D, inner = H * 64;
  const int nthreads = (D / 4 + 31) / 32 * 32;
  int rc = launch_pdl("k_step_embed", k_step_embed, dim3(n), nthreads, 0, 1, st, (const int64_t*)a->ids, (const bf16*)a->embed_real, (const bf16*)a->embed_imag,
                      (const float*)a->embed_scale, w.z, D, a->V, w.best, w.done);
  if (rc) return rc;
  const bf16* delta = nullptr;
  const float* scale = nullptr;
  // the operand of a projection: norm(z + scale * delta) (z in place: only its own row's CTA touches it)
  auto operand = [&](Skinny& p, const float* norm_scale) -> int {
    p.n = n;
    p.K = K2;
    p.x = w.xn;
    return launch_pdl("k_step_norm", k_step_norm, dim3(n), nthreads, 0, 1, st, w.z, delta, scale, norm_scale, w.xn, D);
  };
  for (int l = 0; l < a->n_layers; ++l) {
    const qpam_step_layer& y = a->layers[l];
    Skinny gu{};
    if ((rc = operand(gu, y.n1))) return rc;
    gu.w = (const bf16*)y.w_gu; gu.ld = K2; gu.rows = a->hidden; gu.out = w.gated; gu.act_bias = y.act_bias; gu.act_beta = y.act_beta;
    if ((rc = launch_proj<EPI_GATE>(gu, a->hidden / 8, st))) return rc;
    Skinny dn{};
    dn.n = n; dn.K = 2 * a->hidden; dn.x = w.gated; dn.w = (const bf16*)y.w_down; dn.ld = 2 * a->hidden; dn.rows = D; dn.out = w.delta;
    if ((rc = launch_proj<EPI_COMPLEX>(dn, D / 16, st))) return rc;
    delta = w.delta;
    scale = y.cgu_scale;
    Skinny fr{};
    if ((rc = operand(fr, y.n2))) return rc;
    fr.w = (const bf16*)y.w_front; fr.ld = K2; fr.w2 = (const bf16*)y.w_mag; fr.rows = 3 * inner; fr.rows_a = a->rows_a; fr.rows_m = a->rows_m;
    fr.bias = (const bf16*)y.b_front + 6 * inner; fr.bias2 = (const bf16*)y.b_mag; fr.q = w.q; fr.k = w.k; fr.v = w.v; fr.gates = w.gates;
    fr.rope = a->rope; fr.rope_len = a->rope_len; fr.positions = a->positions; fr.H = H; fr.d = 64; fr.q_scale = a->q_scale;
    if ((rc = launch_proj<EPI_FRONT>(fr, 3 * inner / 16 + (a->rows_a + 15) / 16 + (a->rows_m + 15) / 16, st))) return rc;
    StepRecur sr{};
    sr.pool = a->pool; sr.slots = a->slot_ids; sr.q = w.q; sr.k = w.k; sr.v = w.v; sr.y = w.y; sr.gates = w.gates; sr.dt_bias = y.dt_bias; sr.dt_off = y.dt_off;
    sr.n_slots = a->n_slots; sr.L = a->n_layers; sr.layer = l; sr.H = H; sr.K = a->K; sr.G = a->rows_a + a->rows_m; sr.c_dt = y.col_dt; sr.c_pg = y.col_pg;
    sr.c_phase = a->K > 1 ? y.col_phase : -1; sr.c_score = y.col_score; sr.gamma_floor = y.gamma_floor;
    const dim3 grid(4, H, n);
    rc = a->state_dtype == QPAM_F32 ? launch_pdl("k_step_recur", k_step_recur<float>, grid, 256, 0, 1, st, sr)
                                    : launch_pdl("k_step_recur", k_step_recur<bf16>, grid, 256, 0, 1, st, sr);
    if (rc) return rc;
    Skinny o{};
    o.n = n; o.K = 2 * inner; o.x = w.y; o.w = (const bf16*)y.w_o; o.ld = 2 * inner; o.rows = D; o.out = w.delta;
    if ((rc = launch_proj<EPI_COMPLEX>(o, D / 16, st))) return rc;
    delta = w.delta;
    scale = y.pam_scale;
  }
  Skinny hd{};
  if ((rc = operand(hd, a->out_scale))) return rc;
  bf16* hh = w.delta;                                // (free again: the norm has read it)
  hd.w = (const bf16*)a->w_head; hd.ld = K2; hd.rows = D; hd.bias = (const bf16*)a->b_head; hd.out = hh;
  if ((rc = launch_proj<EPI_COMPLEX>(hd, D / 16, st))) return rc;
  Skinny vo{};
  vo.n = n; vo.K = K2; vo.w = (const bf16*)a->w_vocab; vo.ld = K2; vo.rows = a->V; vo.best = w.best; vo.done = w.done; vo.next_ids = a->next_ids;
  vo.logits = (bf16*)a->logits; vo.ld_logits = a->ld_logits;
  rc = launch_pdl("k_step_norm", k_step_norm, dim3(n), nthreads, 0, 1, st, hh, (const bf16*)nullptr, (const float*)nullptr, (const float*)a->head_norm_scale, w.xn, D);
  if (rc) return rc;
  vo.x = w.xn;
  return launch_vocab(vo, st);
}
