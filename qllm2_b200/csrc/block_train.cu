// Training-step fusions of a V11 block around the library GEMMs and the scan: what the per-operator path runs as ~60
// launches of casts, adds, reductions and element-wise kernels is a few kernels here.
//   k_pack_block / k_unpack_block   every fp32 weight of a block <-> the bf16 matrices its GEMMs read / their gradients
//   k_norm_train                    residual add + norm (+ magnitudes of the normalised rows)
//   k_act_gate_train / _bwd         activation + gated unit; the backward writes the gradient of both projections side by side
//   k_cnorm_res_bwd                 norm backward + the residual's gradient + the scaled branch that was added before it
//   k_front_bwd                     head split, rotary rotation, protect gate, decay and read-out weights, backward, into the
//                                   gradient of ONE projection output (its GEMMs replace four narrow ones and three adds)
//   k_colsum                        all partial parameter gradients of the block
// HBM-bound throughout: a row is read once and written once; parameter gradients stay in registers over the rows a
// thread walks and leave as partial rows.
#include <algorithm>

#include "common.cuh"
#include "elementwise.cuh"

namespace qpam {
namespace {
using namespace ew;
typedef __nv_bfloat16 bf16;

// ------------------------------------------------------------------------------------------------ weights
constexpr int PACK_ITEMS = 24;
struct PackList {
  qpam_pack_item it[PACK_ITEMS];
  int first_block[PACK_ITEMS + 1];
  int n;
};
__device__ __forceinline__ uint2 pack4(float a, float b, float c, float d) {
  const __nv_bfloat162 x = __floats2bfloat162_rn(a, b), y = __floats2bfloat162_rn(c, d);
  return make_uint2(*reinterpret_cast<const uint32_t*>(&x), *reinterpret_cast<const uint32_t*>(&y));
}
__device__ __forceinline__ void unpack8(const uint4& u, float (&r)[4], float (&i)[4]) {      // four interleaved complex values
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    r[j] = __uint_as_float(w[j] << 16);
    i[j] = __uint_as_float(w[j] & 0xffff0000u);
  }
}
__device__ __forceinline__ float2 unpack2(uint32_t w) { return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }

// A CTA takes 256 groups of four source columns of one item.
template <bool UNPACK>
__global__ void __launch_bounds__(256) k_pack_block(const __grid_constant__ PackList L) {
  pdl_wait();
  pdl_trigger();
  int i = 0;
  while (i + 1 < L.n && (int)blockIdx.x >= L.first_block[i + 1]) ++i;
  const qpam_pack_item& t = L.it[i];
  const int64_t g = (int64_t)(blockIdx.x - L.first_block[i]) * 256 + threadIdx.x;
  const int gpr = (t.in + 3) / 4;
  if (g >= (int64_t)t.out * gpr) return;
  const int64_t r = g / gpr;
  const int c = (int)(g - r * gpr) * 4;
  float* a = t.a + r * t.in + c;
  bf16* dst = reinterpret_cast<bf16*>(t.packed);
  if (t.kind == QPAM_PACK_COMPLEX) {          // [2*out][2*in], rows (o, re) = (Wr, -Wi), (o, im) = (Wi, Wr)
    float* b = t.b + r * t.in + c;
    uint4* r0 = reinterpret_cast<uint4*>(dst + 2 * r * (2 * (int64_t)t.in) + 2 * c);
    uint4* r1 = reinterpret_cast<uint4*>(dst + (2 * r + 1) * (2 * (int64_t)t.in) + 2 * c);
    if (!UNPACK) {
      const float4 x = *reinterpret_cast<const float4*>(a), y = *reinterpret_cast<const float4*>(b);
      const uint2 p0 = pack4(x.x, -y.x, x.y, -y.y), p1 = pack4(x.z, -y.z, x.w, -y.w);
      const uint2 q0 = pack4(y.x, x.x, y.y, x.y), q1 = pack4(y.z, x.z, y.w, x.w);
      *r0 = make_uint4(p0.x, p0.y, p1.x, p1.y);
      *r1 = make_uint4(q0.x, q0.y, q1.x, q1.y);
    } else {                                  // dWr = dW[re,re] + dW[im,im],  dWi = dW[im,re] - dW[re,im]
      const uint4 p = *r0, q = *r1;
      const uint32_t pw[4] = {p.x, p.y, p.z, p.w}, qw[4] = {q.x, q.y, q.z, q.w};
      float x[4], y[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 u = unpack2(pw[j]), v = unpack2(qw[j]);
        x[j] = u.x + v.y;
        y[j] = v.x - u.y;
      }
      *reinterpret_cast<float4*>(a) = make_float4(x[0], x[1], x[2], x[3]);
      *reinterpret_cast<float4*>(b) = make_float4(y[0], y[1], y[2], y[3]);
    }
  } else if (t.kind == QPAM_PACK_INTERLEAVE) {  // a Linear over [re | im] planes (in = one plane) <-> interleaved columns
    float* re = t.a + r * 2 * (int64_t)t.in + c;
    float* im = re + t.in;
    uint4* d = reinterpret_cast<uint4*>(dst + r * 2 * (int64_t)t.in + 2 * c);
    if (!UNPACK) {
      const float4 x = *reinterpret_cast<const float4*>(re), y = *reinterpret_cast<const float4*>(im);
      const uint2 p0 = pack4(x.x, y.x, x.y, y.y), p1 = pack4(x.z, y.z, x.w, y.w);
      *d = make_uint4(p0.x, p0.y, p1.x, p1.y);
    } else {
      const uint4 p = *d;
      const float2 u0 = unpack2(p.x), u1 = unpack2(p.y), u2 = unpack2(p.z), u3 = unpack2(p.w);
      *reinterpret_cast<float4*>(re) = make_float4(u0.x, u1.x, u2.x, u3.x);
      *reinterpret_cast<float4*>(im) = make_float4(u0.y, u1.y, u2.y, u3.y);
    }
  } else {                                      // plain rows (a may be null when packing: zeros)
    for (int j = 0; j < 4 && c + j < t.in; ++j) {
      if (!UNPACK) dst[r * t.in + c + j] = __float2bfloat16_rn(t.a ? a[j] : 0.f);
      else a[j] = __bfloat162float(dst[r * t.in + c + j]);
    }
  }
}

// ------------------------------------------------------------------------------------------------ norm
__device__ __forceinline__ float round_bf16(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// z' = z + s delta (delta null: z' = z, not written), xn = norm(z'), mag = |xn|: a warp per row, the row in registers.  The
// arithmetic, its order and every rounding are those of k_scaled_residual_fwd, k_cnorm_fwd and k_cmagnitude in turn.
template <int MAXV>
__global__ void __launch_bounds__(128) k_norm_train(const bf16* __restrict__ z, const bf16* __restrict__ delta, const float* __restrict__ s_ptr,
                                                    const float* __restrict__ scale, bf16* __restrict__ z_out, bf16* __restrict__ xn,
                                                    bf16* __restrict__ mag_out, int64_t N, int D, float eps) {
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x & 31, groups = D >> 2;
  const float s = delta ? *s_ptr : 0.f;
  for (int64_t row = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5); row < N; row += (int64_t)gridDim.x * 4) {
    const int64_t base = row * (int64_t)D * 2;
    float re[MAXV][4], im[MAXV][4], ss = 0.f;
#pragma unroll
    for (int v = 0; v < MAXV; ++v) {
      const int g = v * 32 + lane;
      if (g < groups) {
        V4<bf16>::ld(z + base + g * 8, re[v], im[v]);
        if (delta) {
          float dr[4], di[4];
          V4<bf16>::ld(delta + base + g * 8, dr, di);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            re[v][j] = round_bf16(fmaf(s, dr[j], re[v][j]));
            im[v][j] = round_bf16(fmaf(s, di[j], im[v][j]));
          }
          V4<bf16>::st(z_out + base + g * 8, re[v], im[v]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) ss += re[v][j] * re[v][j] + im[v][j] * im[v][j] + MAG_EPS;
      }
    }
    ss = warp_sum(ss);
    const float rrms = rsqrtf(ss / (float)D + eps);
#pragma unroll
    for (int v = 0; v < MAXV; ++v) {
      const int g = v * 32 + lane;
      if (g < groups) {
        const float4 sc = *reinterpret_cast<const float4*>(scale + g * 4);
        const float s4[4] = {sc.x, sc.y, sc.z, sc.w};
        float m[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const MagInv mag_ = mag_inv(re[v][j] * re[v][j] + im[v][j] * im[v][j] + MAG_EPS);
          const float w = mag_.mag * mag_.inv * rrms * s4[j];
          re[v][j] = round_bf16(re[v][j] * w);
          im[v][j] = round_bf16(im[v][j] * w);
          m[j] = mag_inv(re[v][j] * re[v][j] + im[v][j] * im[v][j] + MAG_EPS).mag;
        }
        V4<bf16>::st(xn + base + g * 8, re[v], im[v]);
        if (mag_out) E4<bf16>::st(mag_out + row * (int64_t)D + g * 4, m);
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------ activation + gate
// out = gate/(|gate|+e) sigmoid(|gate|) * up' (complex), up' = up/(|up|+e) act(|up|) rounded: as k_act_gate, with both
// backward passes of k_cgu_gate_bwd and k_modact_bwd in registers.  dgu [N][gate | up] is one GEMM operand.
template <bool SWISH>
__global__ void __launch_bounds__(512) k_act_gate_train(const bf16* __restrict__ gate, const bf16* __restrict__ up, const float* __restrict__ bias,
                                                        const float* __restrict__ beta, bf16* __restrict__ out, int64_t N, int C) {
  pdl_wait();
  pdl_trigger();
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= (C >> 2)) return;
  float b4[4], be4[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    b4[j] = bias[g * 4 + j];
    be4[j] = SWISH ? beta[g * 4 + j] : 0.f;
  }
#pragma unroll 2
  for (int64_t row = blockIdx.y; row < N; row += gridDim.y) {
    const int64_t at = (row * C + g * 4) * 2;
    float ar[4], ai[4], ur[4], ui[4];
    V4<bf16>::ld(gate + at, ar, ai);
    V4<bf16>::ld(up + at, ur, ui);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const MagInv um = mag_inv(ur[j] * ur[j] + ui[j] * ui[j] + MAG_EPS), gm = mag_inv(ar[j] * ar[j] + ai[j] * ai[j] + MAG_EPS);
      const float act = SWISH ? um.mag * sigmoidf_(be4[j] * um.mag + b4[j]) : fmaxf(um.mag + b4[j], 0.f);
      const float f = act * um.inv;
      const float vr = round_bf16(ur[j] * f), vi = round_bf16(ui[j] * f);
      const float h = sigmoidf_(gm.mag) * gm.inv;
      const float pr = ar[j] * vr - ai[j] * vi, pi = ar[j] * vi + ai[j] * vr;
      ar[j] = pr * h;
      ai[j] = pi * h;
    }
    V4<bf16>::st(out + at, ar, ai);
  }
}

template <bool SWISH>
__global__ void __launch_bounds__(512) k_act_gate_bwd(const bf16* __restrict__ gate, const bf16* __restrict__ up, const bf16* __restrict__ dout,
                                                      const float* __restrict__ bias, const float* __restrict__ beta, bf16* __restrict__ dgu, float* __restrict__ part, int64_t N, int C) {
  pdl_wait();
  pdl_trigger();
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= (C >> 2)) return;
  float b4[4], be4[4], ab[4] = {0.f, 0.f, 0.f, 0.f}, abe[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    b4[j] = bias[g * 4 + j];
    be4[j] = SWISH ? beta[g * 4 + j] : 0.f;
  }
  // the next row is on its way while this one is computed (~100 instructions and six special functions for 20 bytes)
  uint4 na = make_uint4(0u, 0u, 0u, 0u), nu = na, ng = na;
  auto request = [&](int64_t row) {
    if (row >= N) return;
    const int64_t at = (row * C + g * 4) * 2;
    na = *reinterpret_cast<const uint4*>(gate + at);
    nu = *reinterpret_cast<const uint4*>(up + at);
    ng = *reinterpret_cast<const uint4*>(dout + at);
  };
  request(blockIdx.y);
  for (int64_t row = blockIdx.y; row < N; row += gridDim.y) {
    float ar[4], ai[4], ur[4], ui[4], gr[4], gi[4], dr[4], di[4];
    unpack8(na, ar, ai);
    unpack8(nu, ur, ui);
    unpack8(ng, gr, gi);
    request(row + gridDim.y);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const MagInv um = mag_inv(ur[j] * ur[j] + ui[j] * ui[j] + MAG_EPS), gm = mag_inv(ar[j] * ar[j] + ai[j] * ai[j] + MAG_EPS);
      // the activation of `up` and its derivative
      float act, dact, t = 0.f;
      bool on = true;
      if (SWISH) {
        const float s = sigmoidf_(be4[j] * um.mag + b4[j]);
        t = um.mag * s * (1.f - s);
        act = um.mag * s;
        dact = s + t * be4[j];
      } else {
        on = um.mag + b4[j] > 0.f;
        act = on ? um.mag + b4[j] : 0.f;
        dact = on ? 1.f : 0.f;
      }
      const float f = act * um.inv;
      const float vr = round_bf16(ur[j] * f), vi = round_bf16(ui[j] * f);   // up', as the forward rounded it
      // gated unit
      const float sg = sigmoidf_(gm.mag);
      const float h = sg * gm.inv, dh = sg * (1.f - sg) * gm.inv - sg * gm.inv * gm.inv;
      const float pr = ar[j] * vr - ai[j] * vi, pi = ar[j] * vi + ai[j] * vr;
      const float s = gr[j] * pr + gi[j] * pi;
      const float dvr = h * (ar[j] * gr[j] + ai[j] * gi[j]), dvi = h * (ar[j] * gi[j] - ai[j] * gr[j]);
      const float kg = s * dh * gm.rmag;
      dr[j] = h * (vr * gr[j] + vi * gi[j]) + ar[j] * kg;
      di[j] = h * (vr * gi[j] - vi * gr[j]) + ai[j] * kg;
      // back through the activation
      const float q = dvr * ur[j] + dvi * ui[j];
      if (SWISH) {
        ab[j] += q * t * um.inv;
        abe[j] += q * t * um.mag * um.inv;
      } else {
        ab[j] += on ? q * um.inv : 0.f;
      }
      const float ku = q * (dact * um.inv - act * um.inv * um.inv) * um.rmag;
      const float u0 = ur[j], u1 = ui[j];
      ur[j] = dvr * f + u0 * ku;
      ui[j] = dvi * f + u1 * ku;
    }
    bf16* d = dgu + row * (4 * (int64_t)C) + g * 8;
    V4<bf16>::st(d, dr, di);
    V4<bf16>::st(d + 2 * C, ur, ui);
  }
  float* p = part + (int64_t)blockIdx.y * (SWISH ? 2 * C : C) + g * 4;
  *reinterpret_cast<float4*>(p) = make_float4(ab[0], ab[1], ab[2], ab[3]);
  if (SWISH) *reinterpret_cast<float4*>(p + C) = make_float4(abe[0], abe[1], abe[2], abe[3]);
}

// ------------------------------------------------------------------------------------------------ norm + residual
// z' = z + s delta was normalised into xn (whose magnitudes may have been read too); dres is the gradient of z' from the
// residual path.  dz = dres + d(norm) [+ d(|xn|)], ddelta = s dz, partial rows [D + 1] of d(scale) and d(s).
// z here is z' (the stored sum).  Without delta: dz alone.
template <int MAXV>
__global__ void __launch_bounds__(128) k_cnorm_res_bwd(const bf16* __restrict__ z, const float* __restrict__ scale, const bf16* __restrict__ dxn,
                                                       const bf16* __restrict__ dmag, const bf16* __restrict__ dres, const bf16* __restrict__ delta,
                                                       const float* __restrict__ s_ptr, bf16* __restrict__ dz, bf16* __restrict__ ddelta,
                                                       float* __restrict__ part, int64_t N, int D, float eps) {
  pdl_wait();
  pdl_trigger();
  extern __shared__ float sh[];               // [4][D + 1]
  const int lane = threadIdx.x & 31, w4 = threadIdx.x >> 5;
  const int64_t warp = (int64_t)blockIdx.x * 4 + w4, nwarps = (int64_t)gridDim.x * 4;
  const int groups = D >> 2;
  const float s = delta ? *s_ptr : 0.f;
  float acc[MAXV][4], ds = 0.f;
#pragma unroll
  for (int v = 0; v < MAXV; ++v)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[v][j] = 0.f;
  for (int64_t row = warp; row < N; row += nwarps) {
    const int64_t base = row * (int64_t)D * 2;
    // everything the row needs is requested before the first reduction (as it arrives: 16 bytes are eight scalars)
    uint4 zp[MAXV], rp[MAXV], dp[MAXV];
    uint2 mp[MAXV];
    float gr[MAXV][4], gi[MAXV][4], ss = 0.f;
#pragma unroll
    for (int v = 0; v < MAXV; ++v) {
      const int g = v * 32 + lane;
      if (g < groups) {
        zp[v] = *reinterpret_cast<const uint4*>(z + base + g * 8);
        V4<bf16>::ld(dxn + base + g * 8, gr[v], gi[v]);
      }
    }
#pragma unroll
    for (int v = 0; v < MAXV; ++v) {
      const int g = v * 32 + lane;
      rp[v] = dp[v] = make_uint4(0u, 0u, 0u, 0u);
      mp[v] = make_uint2(0u, 0u);
      if (g < groups) {
        if (dres) rp[v] = *reinterpret_cast<const uint4*>(dres + base + g * 8);
        if (dmag) mp[v] = *reinterpret_cast<const uint2*>(dmag + row * (int64_t)D + g * 4);
        if (delta) dp[v] = *reinterpret_cast<const uint4*>(delta + base + g * 8);
      }
    }
#pragma unroll
    for (int v = 0; v < MAXV; ++v)
      if (v * 32 + lane < groups) {
        float re[4], im[4];
        unpack8(zp[v], re, im);
#pragma unroll
        for (int j = 0; j < 4; ++j) ss += re[j] * re[j] + im[j] * im[j] + MAG_EPS;
      }
    ss = warp_sum(ss);
    const float rrms = rsqrtf(ss / (float)D + eps);
    float cs = 0.f;
#pragma unroll
    for (int v = 0; v < MAXV; ++v) {
      const int g = v * 32 + lane;
      if (g < groups) {
        const float4 sc = *reinterpret_cast<const float4*>(scale + g * 4);
        const float s4[4] = {sc.x, sc.y, sc.z, sc.w};
        const float2 m01 = unpack2(mp[v].x), m23 = unpack2(mp[v].y);
        const float dm[4] = {m01.x, m01.y, m23.x, m23.y};
        float re[4], im[4];
        unpack8(zp[v], re, im);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const MagInv m = mag_inv(re[j] * re[j] + im[j] * im[j] + MAG_EPS);
          const float mi = m.mag * m.inv;
          if (dmag) {                         // d|xn| / dxn = xn / |xn| at the rounded xn
            const float wv = mi * rrms * s4[j];
            const float xr = round_bf16(re[j] * wv), xi = round_bf16(im[j] * wv);
            const float q = dm[j] * mag_inv(xr * xr + xi * xi + MAG_EPS).rmag;
            gr[v][j] = fmaf(q, xr, gr[v][j]);
            gi[v][j] = fmaf(q, xi, gi[v][j]);
          }
          cs += (gr[v][j] * re[j] + gi[v][j] * im[j]) * s4[j] * mi;
        }
      }
    }
    cs = warp_sum(cs);
    const float common = cs * rrms * rrms * rrms / (float)D;
#pragma unroll
    for (int v = 0; v < MAXV; ++v) {
      const int g = v * 32 + lane;
      if (g < groups) {
        const float4 sc = *reinterpret_cast<const float4*>(scale + g * 4);
        const float s4[4] = {sc.x, sc.y, sc.z, sc.w};
        float re[4], im[4], rr[4], ri[4];
        unpack8(zp[v], re, im);
        unpack8(rp[v], rr, ri);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const MagInv m = mag_inv(re[j] * re[j] + im[j] * im[j] + MAG_EPS);
          const float mi = m.mag * m.inv;
          const float q = gr[v][j] * re[j] + gi[v][j] * im[j];
          const float wv = mi * rrms * s4[j];
          const float kk = q * s4[j] * MAG_EPS * rrms * m.inv * m.inv * m.rmag - common;
          acc[v][j] += q * mi * rrms;
          rr[j] = round_bf16(rr[j] + gr[v][j] * wv + re[j] * kk);
          ri[j] = round_bf16(ri[j] + gi[v][j] * wv + im[j] * kk);
        }
        V4<bf16>::st(dz + base + g * 8, rr, ri);
        if (delta) {
          float xr[4], xi[4];
          unpack8(dp[v], xr, xi);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            ds = fmaf(rr[j], xr[j], ds);
            ds = fmaf(ri[j], xi[j], ds);
            rr[j] *= s;
            ri[j] *= s;
          }
          V4<bf16>::st(ddelta + base + g * 8, rr, ri);
        }
      }
    }
  }
  ds = warp_sum(ds);
#pragma unroll
  for (int v = 0; v < MAXV; ++v) {
    const int g = v * 32 + lane;
    if (g < groups)
#pragma unroll
      for (int j = 0; j < 4; ++j) sh[w4 * (D + 1) + g * 4 + j] = acc[v][j];
  }
  if (lane == 0) sh[w4 * (D + 1) + D] = ds;
  __syncthreads();
  for (int c = threadIdx.x; c <= D; c += 128)
    part[(int64_t)blockIdx.x * (D + 1) + c] = sh[c] + sh[D + 1 + c] + sh[2 * (D + 1) + c] + sh[3 * (D + 1) + c];
}

// ------------------------------------------------------------------------------------------------ PAM front
// The adjoint of k_pam_front.  A CTA walks tiles of `tile_tok` tokens: threads own (token, head, group of 4 channels) of
// q, k, v; d/4 neighbouring lanes sum a head's Re<dv, v>, which the gate threads -- one (token, head) each -- turn into
// the protect gate's gradient beside the decay's and the read-out weights'.  A tile is as long as the grid allows (28 tokens
// at 16384 tokens): its two barriers and the gates' chain of small loads and transcendentals are paid once for all its
// tokens, while another CTA of the SM streams (112 us with tiles of four tokens, 47 us
// so; 27 us of traffic).
__global__ void __launch_bounds__(1024) k_front_bwd(const __grid_constant__ qpam_front_bwd_args p, int per_tok_pad, int tile_tok) {
  pdl_wait();
  pdl_trigger();
  const qpam_front_args& a = p.f;
  extern __shared__ float domp[];             // [tile_tok][H], then the CTA's sums [tile_tok * H][3K + 1]
  const int H = a.H, K = a.K, d = a.d, gph = d >> 2, tid = threadIdx.x;
  const int64_t ntok = (int64_t)a.B * a.T, ntile = (ntok + tile_tok - 1) / tile_tok;
  const int64_t side = (int64_t)H * d * 2;
  const int slots = blockDim.x / per_tok_pad;   // tokens in flight
  const int my_u = tid / per_tok_pad, idx = tid - my_u * per_tok_pad;
  const bool main_on = my_u < slots && idx < H * gph;
  const int h = main_on ? idx / gph : 0, g = main_on ? idx - h * gph : 0;
  const int NS = 3 * K + 1;
  const bool gate_on = tid < tile_tok * H;
  const int gu = gate_on ? tid / H : 0, gh = gate_on ? tid - gu * H : 0;
  float sx[QPAM_MAX_STATES], sp = 0.f, sph[QPAM_MAX_STATES], ssc[QPAM_MAX_STATES];
#pragma unroll
  for (int k = 0; k < QPAM_MAX_STATES; ++k) sx[k] = sph[k] = ssc[k] = 0.f;
  bf16* draw = reinterpret_cast<bf16*>(p.d_raw);
  bf16* drawm = reinterpret_cast<bf16*>(p.d_rawm);
  for (int64_t tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
    for (int u0 = 0; u0 < tile_tok; u0 += slots) {
      const int u = u0 + my_u;
      const int64_t tok = tile * tile_tok + u;
      const bool on = main_on && u < tile_tok && tok < ntok;
      float dot = 0.f;
      if (on) {
        const int b = (int)(tok / a.T), t = (int)(tok - (int64_t)b * a.T);
        const int64_t src = (((int64_t)b * H + h) * a.T + t) * (int64_t)d * 2 + g * 8;
        float re[3][4], im[3][4], vr[4], vi[4];
        V4<bf16>::ld(reinterpret_cast<const bf16*>(a.q) + src, re[0], im[0]);
        V4<bf16>::ld(reinterpret_cast<const bf16*>(a.k) + src, re[1], im[1]);
        V4<bf16>::ld(reinterpret_cast<const bf16*>(a.v) + src, re[2], im[2]);
        V4<bf16>::ld(reinterpret_cast<const bf16*>(a.qkv) + tok * a.ld_qkv + 2 * side + (int64_t)h * d * 2 + g * 8, vr, vi);
        const float keep = a.pg ? 1.f - sigmoidf_(__bfloat162float(reinterpret_cast<const bf16*>(a.pg)[tok * a.ld_pg + h])) : 1.f;
        float4 c0 = make_float4(1.f, 0.f, 1.f, 0.f), c1 = c0;
        if (a.rope) {
          int64_t pos = a.positions ? a.positions[tok] : a.offset + t;
          pos = pos < 0 ? 0 : (pos >= a.rope_len ? a.rope_len - 1 : pos);
          c0 = *reinterpret_cast<const float4*>(a.rope + (pos * d + g * 4) * 2);
          c1 = *reinterpret_cast<const float4*>(a.rope + (pos * d + g * 4) * 2 + 4);
        }
        const float cs[4] = {c0.x, c0.z, c1.x, c1.z}, sn[4] = {c0.y, c0.w, c1.y, c1.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          dot += vr[j] * re[2][j] + vi[j] * im[2][j];
#pragma unroll
          for (int w = 0; w < 2; ++w) {       // the gradient rotates back
            const float m = w == 0 ? a.q_scale : 1.f, r0 = re[w][j], i0 = im[w][j];
            re[w][j] = (r0 * cs[j] + i0 * sn[j]) * m;
            im[w][j] = (i0 * cs[j] - r0 * sn[j]) * m;
          }
          re[2][j] *= keep;
          im[2][j] *= keep;
        }
        bf16* dst = draw + tok * p.ld_raw + (int64_t)h * d * 2 + g * 8;
#pragma unroll
        for (int w = 0; w < 3; ++w) V4<bf16>::st(dst + w * side, re[w], im[w]);
      }
      for (int o = gph >> 1; o; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
      if (on && g == 0) domp[u * H + h] = dot;
    }
    __syncthreads();
    const int64_t tok = tile * tile_tok + gu;
    if (gate_on && tok < ntok) {
      const int b = (int)(tok / a.T), t = (int)(tok - (int64_t)b * a.T);
      const float dtv = __bfloat162float(reinterpret_cast<const bf16*>(a.dt)[tok * a.ld_dt + gh]) + a.dt_bias[gh];
      const float pr = a.pg ? sigmoidf_(__bfloat162float(reinterpret_cast<const bf16*>(a.pg)[tok * a.ld_pg + gh])) : 0.f;
      float w[QPAM_MAX_STATES], dw[QPAM_MAX_STATES], wmax = -INFINITY, wsum = 0.f, wdw = 0.f, dp = 0.f, ddt = 0.f;
#pragma unroll
      for (int k = 0; k < QPAM_MAX_STATES; ++k) w[k] = 1.f;
      if (a.score) {
        const bf16* sc = reinterpret_cast<const bf16*>(a.score) + tok * a.ld_score + gh * K;
        for (int k = 0; k < K; ++k) wmax = fmaxf(wmax, __bfloat162float(sc[k]));
#pragma unroll
        for (int k = 0; k < QPAM_MAX_STATES; ++k)
          if (k < K) { w[k] = __expf(__bfloat162float(sc[k]) - wmax); wsum += w[k]; }
#pragma unroll
        for (int k = 0; k < QPAM_MAX_STATES; ++k) w[k] = w[k] / wsum * (float)K;
      }
      auto out = [&](int which, int i, float v) {
        if (p.col[which] >= 0) (p.from_mag[which] ? drawm + tok * p.ld_rawm : draw + tok * p.ld_raw)[p.col[which] + i] = __float2bfloat16_rn(v);
      };
#pragma unroll
      for (int k = 0; k < QPAM_MAX_STATES; ++k)
        if (k < K) {
          const float x = dtv + (a.state_dt_offset ? a.state_dt_offset[k] : 0.f);
          const float base = sigmoidf_(-x);
          const float basef = a.gamma_floor > 0.f ? a.gamma_floor + (1.f - a.gamma_floor) * base : base;
          const int64_t gi = (((int64_t)k * a.B + b) * H + gh) * a.T + t;
          const float dg = a.gamma[gi];
          dp += dg * (1.f - basef);
          const float dx = -(1.f - (a.gamma_floor > 0.f ? a.gamma_floor : 0.f)) * dg * (1.f - pr) * base * (1.f - base);
          ddt += dx;
          sx[k] += dx;
          dw[k] = 0.f;
          if (a.coef && a.phase) {
            float sn, cs;
            sincosf(__bfloat162float(reinterpret_cast<const bf16*>(a.phase)[tok * a.ld_phase + gh * K + k]), &sn, &cs);
            const float2 dc = *reinterpret_cast<const float2*>(a.coef + gi * 2);
            dw[k] = cs * dc.x + sn * dc.y;
            const float dph = w[k] * (cs * dc.y - sn * dc.x);
            sph[k] += dph;
            out(2, gh * K + k, dph);
            wdw += w[k] * dw[k];
          }
        }
      out(0, gh, ddt);
      if (a.pg) {
        const float v = (dp - domp[gu * H + gh]) * pr * (1.f - pr);
        sp += v;
        out(1, gh, v);
      }
      if (a.score) {
#pragma unroll
        for (int k = 0; k < QPAM_MAX_STATES; ++k)
          if (k < K) {
            const float v = w[k] * (dw[k] - wdw / (float)K);
            ssc[k] += v;
            out(3, gh * K + k, v);
          }
      }
      if (gh == 0) {                           // padding columns of both projections
        for (int c = p.used_raw; c < p.ld_raw; ++c) draw[tok * p.ld_raw + c] = __float2bfloat16_rn(0.f);
        if (drawm)
          for (int c = p.used_rawm; c < p.ld_rawm; ++c) drawm[tok * p.ld_rawm + c] = __float2bfloat16_rn(0.f);
      }
    }
    __syncthreads();
  }
  // sums over this CTA's tokens: column (h, .) of [dx_k | dpg | dphase_k | dscore_k], rows in order
  if (gate_on) {
    float* s = domp + tid * NS;
#pragma unroll
    for (int k = 0; k < QPAM_MAX_STATES; ++k)
      if (k < K) { s[k] = sx[k]; s[K + 1 + k] = sph[k]; s[2 * K + 1 + k] = ssc[k]; }
    s[K] = sp;
  }
  __syncthreads();
  for (int c = tid; c < H * NS; c += blockDim.x) {
    float v = 0.f;
    const int hh = c / NS, i = c - hh * NS;
    for (int u = 0; u < tile_tok; ++u) v += domp[(u * H + hh) * NS + i];
    p.part[(int64_t)blockIdx.x * H * NS + c] = v;
  }
}

// ------------------------------------------------------------------------------------------------ column sums
constexpr int SUM_ITEMS = 12;
struct SumList {
  qpam_colsum_item it[SUM_ITEMS];
  int first_block[SUM_ITEMS + 1];
  int n;
};
// out[c] = sum_p part[p][c]; a CTA takes 32 columns, 32 threads each.
__global__ void __launch_bounds__(1024) k_colsum(const __grid_constant__ SumList L) {
  pdl_wait();
  pdl_trigger();
  __shared__ float sh[32][33];
  int i = 0;
  while (i + 1 < L.n && (int)blockIdx.x >= L.first_block[i + 1]) ++i;
  const qpam_colsum_item& t = L.it[i];
  const int c = (blockIdx.x - L.first_block[i]) * 32 + (threadIdx.x & 31), r = threadIdx.x >> 5;
  float v = 0.f;
  if (c < t.C) {
#pragma unroll 4
    for (int p = r; p < t.P; p += 32) v += t.part[(int64_t)p * t.ld + c];
  }
  sh[r][threadIdx.x & 31] = v;
  __syncthreads();
  if (r == 0 && c < t.C) {
    float s = 0.f;
#pragma unroll
    for (int q = 0; q < 32; ++q) s += sh[q][threadIdx.x];
    t.out[c] = s;
  }
}

// Parameter gradients of the front from the sums [H][3K+1] of d(x_k), d(pg), d(phase_k), d(score_k).
__global__ void k_front_params(const float* __restrict__ s, int H, int K, float* dt_bias, float* dt_proj_bias, float* dt_off, float* pg, float* phase,
                               float* score) {
  const int NS = 3 * K + 1;
  for (int h = threadIdx.x; h < H; h += blockDim.x) {
    float v = 0.f;
    for (int k = 0; k < K; ++k) {
      v += s[h * NS + k];
      if (phase) phase[h * K + k] = s[h * NS + K + 1 + k];
      if (score) score[h * K + k] = s[h * NS + 2 * K + 1 + k];
    }
    dt_bias[h] = v;
    dt_proj_bias[h] = v;
    if (pg) pg[h] = s[h * NS + K];
  }
  if (dt_off && threadIdx.x < K) {
    float v = 0.f;
    for (int h = 0; h < H; ++h) v += s[h * NS + threadIdx.x];
    dt_off[threadIdx.x] = v;
  }
}

template <bool UNPACK>
int pack_launch(const qpam_pack_item* items, int32_t n, void* stream) {
  QPAM_REQUIRE(items && n >= 1 && n <= PACK_ITEMS, "pack_block: 1..%d items (got %d)", PACK_ITEMS, n);
  PackList L{};
  L.n = n;
  int blocks = 0;
  for (int i = 0; i < n; ++i) {
    const qpam_pack_item& t = items[i];
    QPAM_REQUIRE(t.packed && t.out > 0 && t.in > 0 && t.kind >= 0 && t.kind <= QPAM_PACK_PLAIN, "pack_block: bad item %d", i);
    QPAM_REQUIRE((t.a || (!UNPACK && t.kind == QPAM_PACK_PLAIN)) && (t.b || t.kind != QPAM_PACK_COMPLEX), "pack_block: NULL pointer in item %d", i);
    QPAM_REQUIRE(t.kind == QPAM_PACK_PLAIN || t.in % 4 == 0, "pack_block: in must be a multiple of 4 (item %d)", i);
    L.it[i] = t;
    L.first_block[i] = blocks;
    blocks += (int)(((int64_t)t.out * ((t.in + 3) / 4) + 255) / 256);
  }
  L.first_block[n] = blocks;
  cudaStream_t st = (cudaStream_t)stream;
  launch_after(k_pack_block<UNPACK>, blocks, 256, 0, st, L);
  QPAM_LAUNCH_CHECK("k_pack_block");
  return QPAM_OK;
}

}  // namespace
}  // namespace qpam

using namespace qpam;
using namespace qpam::ew;

extern "C" int qpam_pack_block(const qpam_pack_item* items, int32_t n, void* stream) { return pack_launch<false>(items, n, stream); }
extern "C" int qpam_unpack_block(const qpam_pack_item* items, int32_t n, void* stream) { return pack_launch<true>(items, n, stream); }

extern "C" int qpam_colsum(const qpam_colsum_item* items, int32_t n, void* stream) {
  QPAM_REQUIRE(items && n >= 1 && n <= SUM_ITEMS, "colsum: 1..%d items (got %d)", SUM_ITEMS, n);
  SumList L{};
  L.n = n;
  int blocks = 0;
  for (int i = 0; i < n; ++i) {
    QPAM_REQUIRE(items[i].part && items[i].out && items[i].P > 0 && items[i].C > 0 && items[i].ld >= items[i].C, "colsum: bad item %d", i);
    L.it[i] = items[i];
    L.first_block[i] = blocks;
    blocks += (items[i].C + 31) / 32;
  }
  L.first_block[n] = blocks;
  cudaStream_t st = (cudaStream_t)stream;
  launch_after(k_colsum, blocks, 1024, 0, st, L);
  QPAM_LAUNCH_CHECK("k_colsum");
  return QPAM_OK;
}

extern "C" int qpam_norm_train_fwd(const void* z, const void* delta, const float* s, const float* scale, void* z_out, void* xn, void* mag, int64_t N,
                                   int32_t D, float eps, void* stream) {
  QPAM_REQUIRE(z && scale && xn && (!delta || (s && z_out)), "norm_train: NULL pointer argument");
  QPAM_REQUIRE(N > 0 && D > 0 && D % 4 == 0 && D <= 768, "norm_train: D must be a multiple of 4 up to 768 (got %d)", D);
  cudaStream_t st = (cudaStream_t)stream;
  const int blocks = (int)std::min<int64_t>((N + 3) / 4, sm_count() * 16);
#define QPAM_NT(MV) \
  launch_after(k_norm_train<MV>, blocks, 128, 0, st, (const bf16*)z, (const bf16*)delta, s, scale, (bf16*)z_out, (bf16*)xn, (bf16*)mag, N, D, eps)
  if (D <= 384) QPAM_NT(3);
  else QPAM_NT(6);
#undef QPAM_NT
  QPAM_LAUNCH_CHECK("k_norm_train");
  return QPAM_OK;
}

extern "C" int qpam_act_gate_train_fwd(const void* gate, const void* up, const float* bias, const float* beta, void* out, int64_t N, int32_t C, void* stream) {
  QPAM_REQUIRE(gate && up && bias && out, "act_gate_train: NULL pointer argument");
  QPAM_REQUIRE(N > 0 && C > 0 && C % 4 == 0, "act_gate_train: C must be a multiple of 4 (got %d)", C);
  cudaStream_t st = (cudaStream_t)stream;
  const int groups = C / 4, threads = pick_threads(groups), xb = (groups + threads - 1) / threads;
  dim3 grid(xb, (unsigned)std::min<int64_t>(N, std::max(1, (sm_count() * 2048) / (xb * threads))));
  if (beta) launch_after(k_act_gate_train<true>, grid, threads, 0, st, (const bf16*)gate, (const bf16*)up, bias, beta, (bf16*)out, N, C);
  else launch_after(k_act_gate_train<false>, grid, threads, 0, st, (const bf16*)gate, (const bf16*)up, bias, beta, (bf16*)out, N, C);
  QPAM_LAUNCH_CHECK("k_act_gate_train");
  return QPAM_OK;
}

extern "C" int32_t qpam_act_gate_bwd_parts(int64_t N, int32_t C) {
  const int groups = C / 4, threads = pick_threads(groups), xb = (groups + threads - 1) / threads;
  return (int32_t)std::max<int64_t>(1, std::min<int64_t>(N, (int64_t)sm_count() * 1536 / (xb * threads)));
}
extern "C" int qpam_act_gate_bwd(const void* gate, const void* up, const void* dout, const float* bias, const float* beta, void* dgate_up, float* part, int32_t P,
                                 int64_t N, int32_t C, void* stream) {
  QPAM_REQUIRE(gate && up && dout && bias && dgate_up && part, "act_gate_bwd: NULL pointer argument");
  QPAM_REQUIRE(N > 0 && C > 0 && C % 4 == 0 && P > 0 && P <= 65535, "act_gate_bwd: bad sizes (C must be a multiple of 4)");
  cudaStream_t st = (cudaStream_t)stream;
  const int groups = C / 4, threads = pick_threads(groups);
  dim3 grid((groups + threads - 1) / threads, P);
  if (beta) launch_after(k_act_gate_bwd<true>, grid, threads, 0, st, (const bf16*)gate, (const bf16*)up, (const bf16*)dout, bias, beta, (bf16*)dgate_up, part, N, C);
  else launch_after(k_act_gate_bwd<false>, grid, threads, 0, st, (const bf16*)gate, (const bf16*)up, (const bf16*)dout, bias, beta, (bf16*)dgate_up, part, N, C);
  QPAM_LAUNCH_CHECK("k_act_gate_bwd");
  return QPAM_OK;
}

extern "C" int qpam_cnorm_res_bwd(const void* z, const float* scale, const void* dxn, const void* dmag, const void* dres, const void* delta, const float* s,
                                  void* dz, void* ddelta, float* part, int32_t P, int64_t N, int32_t D, float eps, void* stream) {
  QPAM_REQUIRE(z && scale && dxn && dz && part && (!delta || (s && ddelta)), "cnorm_res_bwd: NULL pointer argument");
  QPAM_REQUIRE(N > 0 && D > 0 && D % 4 == 0 && D <= 768 && P > 0, "cnorm_res_bwd: D must be a multiple of 4 up to 768 (got %d)", D);
  cudaStream_t st = (cudaStream_t)stream;
  const size_t smem = (size_t)4 * (D + 1) * sizeof(float);
#define QPAM_NRB(MV)                                                                                                                      \
  launch_after(k_cnorm_res_bwd<MV>, P, 128, smem, st, (const bf16*)z, scale, (const bf16*)dxn, (const bf16*)dmag, (const bf16*)dres, (const bf16*)delta, s, \
                                            (bf16*)dz, (bf16*)ddelta, part, N, D, eps)
  if (D <= 384) QPAM_NRB(3);
  else QPAM_NRB(6);
#undef QPAM_NRB
  QPAM_LAUNCH_CHECK("k_cnorm_res_bwd");
  return QPAM_OK;
}

extern "C" int qpam_pam_front_bwd(const qpam_front_bwd_args* p, void* stream) {
  QPAM_REQUIRE(p && p->f.qkv && p->f.dt && p->f.dt_bias && p->f.q && p->f.k && p->f.v && p->f.gamma && p->d_raw && p->part, "front_bwd: NULL pointer argument");
  const qpam_front_args& a = p->f;
  QPAM_REQUIRE(a.io_dtype == QPAM_BF16 && a.B > 0 && a.T > 0 && a.H > 0 && a.H <= 64 && a.K >= 1 && a.K <= QPAM_MAX_STATES, "front_bwd: bad dtype or shape");
  QPAM_REQUIRE(a.d >= 4 && a.d <= 128 && (a.d & (a.d - 1)) == 0, "front_bwd: head_dim must be a power of two in [4,128]");
  QPAM_REQUIRE(p->P > 0 && p->ld_raw >= 6 * (int64_t)a.H * a.d && p->ld_raw % 8 == 0, "front_bwd: bad output rows");
  for (int i = 0; i < 4; ++i) QPAM_REQUIRE(p->col[i] < 0 || !p->from_mag[i] || p->d_rawm, "front_bwd: gate columns without their buffer");
  const int per_tok = (a.H * (a.d / 4) + 31) / 32 * 32;
  QPAM_REQUIRE(per_tok <= 1024, "front_bwd: H * d too large");
  const int slots = std::max(1, std::min(4, 384 / per_tok));        // tokens in flight
  const int threads = std::max(per_tok * slots, (slots * a.H + 31) / 32 * 32);
  const int64_t share = ((int64_t)a.B * a.T + p->P - 1) / p->P;
  const int most = std::max(slots, std::min(threads, 900) / a.H / slots * slots);     // a gate thread per (token, head); 48 KB of sums
  const int tile = (int)std::min<int64_t>(most, (share + slots - 1) / slots * slots);
  const size_t smem = (size_t)tile * a.H * (3 * a.K + 1) * sizeof(float);
  cudaStream_t st = (cudaStream_t)stream;
  launch_after(k_front_bwd, p->P, threads, smem, st, *p, per_tok, tile);
  QPAM_LAUNCH_CHECK("k_front_bwd");
  return QPAM_OK;
}

extern "C" int qpam_front_params(const float* sums, int32_t H, int32_t K, float* dt_bias, float* dt_proj_bias, float* dt_off, float* pg_bias,
                                 float* phase_bias, float* score_bias, void* stream) {
  QPAM_REQUIRE(sums && dt_bias && dt_proj_bias && H > 0 && K >= 1 && K <= QPAM_MAX_STATES, "front_params: bad arguments");
  cudaStream_t st = (cudaStream_t)stream;
  k_front_params<<<1, 64, 0, st>>>(sums, H, K, dt_bias, dt_proj_bias, dt_off, pg_bias, phase_bias, score_bias);
  QPAM_LAUNCH_CHECK("k_front_params");
  return QPAM_OK;
}
