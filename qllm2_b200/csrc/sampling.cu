// Token sampling on the device: temperature, repetition penalty, top-k, top-p (nucleus) and the draw itself,
// one CTA per row of logits, no sort and no host round trip.  Semantics of the reference's sampling block
// (v11/model.py:1221-1244):
//   x = logits / temperature
//   x[h] = x[h] > 0 ? x[h] / penalty : x[h] * penalty          for every token h already in the sequence
//   top-k : drop x < (k-th largest x)                            (ties with the k-th value stay)
//   top-p : in descending order, drop a token when the probability mass BEFORE it is >= top_p
//   draw from softmax of what is left
// The draw is the inverse CDF in vocabulary order of a uniform number the caller supplies.  Nothing depends on the
// order of atomics, so the same inputs give the same token on every run.  Tokens that tie with the nucleus threshold are
// all kept (a sort would keep an arbitrary subset of them).
//
// What bounds it: the row is 100 KB (bf16, V = 50 k) and the 256 rows of a full engine are 26 MB, 4 us of HBM.  A row is never
// copied: every pass streams it again with 16-byte loads (L1 / L2 hits after the first), which leaves room for two CTAs per
// SM, and what a pass costs is its instructions for 98 elements a thread.  So a pass does per element only what it must:
//   * the tokens of the penalty are one bit each in shared memory.  A pass drops them (-inf in the raw word) and takes them one
//     by one afterwards, warp by warp for the warp's own stretch: some lane of a warp holds one in nine of ten steps, and the
//     division and its tests for eight elements were then most of the pass;
//   * the maximum is taken on the raw (packed) values, scaled once per block of four groups;
//   * a comparison with a bin's rough edges decides for nearly every element whether its bin has to be formed at all.
//   small top-k   pass 1 leaves the largest value of every block of four groups (32 or 16 values); the k-th largest of the
//                 threads' maxima is a lower bound of the k-th largest of the row, so only blocks that reach it (about k) are
//                 read again, a group for each thread; the values at or above the bound (about k + k^2 / threads) are a list
//                 and everything after that works on that list: ranks by counting, no search.
//   otherwise     counts or probability mass over 2048 bins LINEAR in x (leading bits of the float pattern put most of a
//                 row into a dozen bins, whose atomics serialise), the bin in which the k-th value / the nucleus closes,
//                 and the exact threshold from the elements of that bin.  Masses are accumulated in fixed point: the
//                 sums do not depend on the order of the atomics.
// Launched with programmatic overlap (it waits at its top): 256 rows behind one another 21.3 -> 19.7 us.
// 256 rows x 50261 bf16 logits with a penalty over 16..513 tokens (captured calls back to back): top-k 50 + top-p 0.9 33.7 -> 20.4 us;
// top-p 0.9 alone 121 -> 78; neither 51.9 -> 28.6.  One row: 17.2 -> 15.2, 58.3 -> 47.8, 22.9 -> 18.5.  (Before: eight tests and a
// division for every group of a pass, the small top-k reading the whole row twice, one warp walking the stretch of the draw.)
#include "common.cuh"
#include "elementwise.cuh"

namespace qpam {
namespace {

constexpr int SAMPLE_LIST = 1024;            // values that the list steps can hold
constexpr int SAMPLE_LIST_TOP_K = 384;       // top-k up to which the list is expected to fit (512 threads: ~710 values)
constexpr int SAMPLE_BINS = 2048;
constexpr int SAMPLE_BLOCKS = 4096;          // blocks of a row (several of a thread's steps share one when a row has more)
constexpr int SAMPLE_ITEMS = 2048;
constexpr float SAMPLE_BINS_PER_UNIT = 64.f;  // bins reach 32 units below the maximum (e^-32 of its mass)
constexpr size_t SAMPLE_SMEM_BITMAP = 160 * 1024;

struct SampleParams {
  const void* logits;
  int64_t ldl;
  const int32_t* slot_ids;
  int64_t* history;
  int64_t ld_hist;
  int32_t* hist_len;
  const float* uniforms;
  int64_t* next_ids;
  float* stats;
  uint32_t* bitmaps;      // [n][words] in the workspace when a bitmap does not fit in shared memory
  int32_t n, V, n_hist_rows, hist_cols, top_k, append, bitmap_words;
  int32_t mass_half;      // masses are integers of 2 * mass_half bits; V sums of one half fit 32 bits
  float inv_temperature, top_p, penalty;
};

__device__ __forceinline__ uint32_t order_key(float x) {
  const uint32_t u = __float_as_uint(x);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_value(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

struct Scratch {
  union {
    uint32_t bins[3][SAMPLE_BINS];     // counts | low and high half of the masses
    struct {
      float top[SAMPLE_BLOCKS];        // [block][thread] largest value of a block
      int item[SAMPLE_ITEMS];          // blocks to read again
    } blocks;
    struct {
      float e[SAMPLE_LIST];            // survivors of top-k in vocabulary order
      int idx[SAMPLE_LIST];
    } sorted;
  };
  uint32_t key[SAMPLE_LIST];           // collected values (any order); 0 = none
  int idx[SAMPLE_LIST];
  double warp_d[32];
  float warp_f[32];
  int n_list, n_item, cross_bin, chosen, last_kept, warp_i[32];
  double cross_before;
  uint32_t limit;
};

template <int NT>
__device__ __forceinline__ float block_max(float v, Scratch* sc) {
  for (int o = 16; o; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sc->warp_f[threadIdx.x >> 5] = v;
  __syncthreads();
  float r = sc->warp_f[threadIdx.x & (NT / 32 - 1)];
  for (int o = NT / 64; o; o >>= 1) r = fmaxf(r, __shfl_xor_sync(0xffffffffu, r, o));
  return r;
}

template <int NT>
__device__ __forceinline__ double block_sum(double v, Scratch* sc) {
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sc->warp_d[threadIdx.x >> 5] = v;
  __syncthreads();
  double r = sc->warp_d[threadIdx.x & (NT / 32 - 1)];
  for (int o = NT / 64; o; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
  return r;
}

// The row as groups of 16 aligned bytes.  Group g holds the elements [g * VEC - lead, (g + 1) * VEC - lead): rows need
// not start on a 16-byte boundary; the first and last group are read element by element, with -inf outside the row.
template <typename T>
struct Row {
  static constexpr int VEC = 16 / (int)sizeof(T);
  const T* base;
  const uint32_t* bits;    // penalised elements by shifted position (index + lead); null = none
  int V, lead, groups;
  float inv_t, penalty;
  bool flat;               // infinite temperature: every finite logit is 0

  __device__ __forceinline__ void init(const T* row, int V_) {
    base = row;
    V = V_;
    lead = (int)((reinterpret_cast<uintptr_t>(row) & 15u) / sizeof(T));
    groups = (V + lead + VEC - 1) / VEC;
  }
  __device__ __forceinline__ uint4 raw(int g) const {
    const int i0 = g * VEC - lead;
    if (i0 >= 0 && i0 + VEC <= V && !flat) return __ldg(reinterpret_cast<const uint4*>(base + i0));
    union { uint4 u; T t[VEC]; } r;
    const uint32_t none = sizeof(T) == 2 ? 0xff80ff80u : 0xff800000u;      // -inf
    r.u = make_uint4(none, none, none, none);
#pragma unroll
    for (int j = 0; j < VEC; ++j)
      if (i0 + j >= 0 && i0 + j < V) r.t[j] = flat ? (T)((float)base[i0 + j] * 0.f) : base[i0 + j];
    return r.u;
  }
  __device__ __forceinline__ uint32_t marks(int g) const {      // one bit for each element of a group (a word holds whole groups)
    const int s = g * VEC;
    return (bits[s >> 5] >> (s & 31)) & ((1u << VEC) - 1u);
  }
  // the group with -inf for its penalised elements
  __device__ __forceinline__ uint4 plain(int g, uint4 u) const {
    if (bits == nullptr) return u;
    const uint32_t m = marks(g);
    if (m == 0u) return u;
    uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if constexpr (sizeof(T) == 2) {
        if (m >> (2 * j) & 1u) w[j] = (w[j] & 0xffff0000u) | 0xff80u;
        if (m >> (2 * j + 1) & 1u) w[j] = (w[j] & 0xffffu) | 0xff800000u;
      } else {
        if (m >> j & 1u) w[j] = 0xff800000u;
      }
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
  }
  // divided by the temperature
  __device__ __forceinline__ void scaled(uint4 u, float (&x)[VEC]) const {
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if constexpr (sizeof(T) == 2) {
        x[2 * j] = __uint_as_float(w[j] << 16) * inv_t;
        x[2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u) * inv_t;
      } else {
        x[j] = __uint_as_float(w[j]) * inv_t;
      }
    }
  }
  __device__ __forceinline__ float penalised(float x) const { return x > 0.f ? x / penalty : x * penalty; }
  __device__ __forceinline__ float penalised_at(int i) const {
    return penalised((float)base[i] * (flat ? 0.f : inv_t));
  }
  // temperature and penalty, in vocabulary order
  __device__ __forceinline__ void values(int g, uint4 u, float (&x)[VEC]) const {
    scaled(u, x);
    if (bits) {
      const uint32_t m = marks(g);
      if (m) {
#pragma unroll
        for (int j = 0; j < VEC; ++j)
          if (m >> j & 1u) x[j] = penalised(x[j]);
      }
    }
  }
};

// Running maximum of raw groups, a NaN losing to any number.
template <typename T>
struct RawMax;
template <>
struct RawMax<float> {
  float m = -INFINITY;
  __device__ __forceinline__ void add(uint4 u) {
    m = fmaxf(fmaxf(m, fmaxf(__uint_as_float(u.x), __uint_as_float(u.y))), fmaxf(__uint_as_float(u.z), __uint_as_float(u.w)));
  }
  __device__ __forceinline__ float value() const { return m; }
};
template <>
struct RawMax<__nv_bfloat16> {
  uint32_t m = 0xff80ff80u;
  static __device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b) {
    const __nv_bfloat162 r = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
    return *reinterpret_cast<const uint32_t*>(&r);
  }
  __device__ __forceinline__ void add(uint4 u) { m = max2(m, max2(max2(u.x, u.y), max2(u.z, u.w))); }
  __device__ __forceinline__ float value() const { return fmaxf(__uint_as_float(m << 16), __uint_as_float(m & 0xffff0000u)); }
};

// Every warp walks its own contiguous stretch of the row, four groups in flight per lane; f(index, x) for one element after another.
// EXACT: every element in its place.  Otherwise the penalised elements are -inf there and come one by one afterwards
// (for_marked), for the warp's own stretch.
template <int NT, typename T, typename F>
__device__ __forceinline__ void for_marked(const Row<T>& r, F one) {
  if (r.bits == nullptr) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int per = (r.groups + NT / 32 - 1) / (NT / 32);
  const int s0 = warp * per * Row<T>::VEC, s1 = min(r.groups, (warp + 1) * per) * Row<T>::VEC;      // shifted positions
  for (int w = (s0 >> 5) + lane; w * 32 < s1; w += 32) {
    uint32_t m = r.bits[w];
    if (w * 32 < s0) m &= ~0u << (s0 & 31);
    if (s1 - w * 32 < 32) m &= (1u << (s1 & 31)) - 1u;
    while (m) {
      const int i = w * 32 + __ffs((int)m) - 1 - r.lead;
      m &= m - 1;
      one(i, r.penalised_at(i));
    }
  }
}
template <int NT, bool EXACT, typename T, typename F>
__device__ __forceinline__ void for_each(const Row<T>& r, F f) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int per = (r.groups + NT / 32 - 1) / (NT / 32);
  const int g1 = min(r.groups, (warp + 1) * per);
  for (int g = warp * per + lane; g < g1; g += 128) {
    uint4 u[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (g + 32 * k < g1) u[k] = r.raw(g + 32 * k);
#pragma unroll 1
    for (int gk = g; gk < min(g1, g + 128); gk += 32) {
      const uint4 c = EXACT ? u[0] : r.plain(gk, u[0]);
      u[0] = u[1]; u[1] = u[2]; u[2] = u[3];
      float x[Row<T>::VEC];
      if (EXACT) r.values(gk, c, x);
      else r.scaled(c, x);
      const int i0 = gk * Row<T>::VEC - r.lead;
#pragma unroll
      for (int j = 0; j < Row<T>::VEC; ++j) f(i0 + j, x[j]);
    }
  }
}

__device__ __forceinline__ void list_add(Scratch* sc, uint32_t key, int i) {
  const int at = atomicAdd(&sc->n_list, 1);
  if (at < SAMPLE_LIST) {
    sc->key[at] = key;
    sc->idx[at] = i;
  }
}

__device__ __forceinline__ int bin_of(float x, float mx) {      // (the conversion saturates: below zero and NaN give 0)
  return (int)min(__float2uint_rz(fmaf(x, -SAMPLE_BINS_PER_UNIT, mx * SAMPLE_BINS_PER_UNIT)), (uint32_t)(SAMPLE_BINS - 1));
}
// Unnormalised probability e^(x - mx): fp32 with gradual underflow, so a token counts (and can be drawn) down to about 103 below the
// maximum.
__device__ __forceinline__ float mass_of(float x, float mx) { return ew::fexp_gradual_(x - mx); }
// The same where it is only a term of a sum that also holds the maximum's 1: results below 2^-126 are zero, as they vanish in such
// a sum.  (Top-p without top-k is 5 % faster for it.  With it everywhere a row without filters takes 27.4 us, not 28.6, and loses
// its tokens beyond 87.)
__device__ __forceinline__ float mass_term(float x, float mx) { return ew::fexp_(x - mx); }
// What few elements of a pass need stays out of line: 32 copies of it in a loop that jumps over them cost more than the pass.
__device__ __noinline__ void list_bin_value(Scratch* sc, float x, float mx, int i, int cross, uint32_t key_k) {
  if (bin_of(x, mx) != cross || order_key(x) < key_k) return;
  const float e = mass_of(x, mx);
  if (e > 0.f) list_add(sc, __float_as_uint(e), i);
}
// unnormalised probability of a kept value, 0 for a dropped one
__device__ __forceinline__ float kept_mass_of(float x, float mx, int cross, uint32_t e_min, uint32_t key_k) {
  const float e = order_key(x) >= key_k ? mass_of(x, mx) : 0.f;
  if (cross < SAMPLE_BINS) {
    const int b = bin_of(x, mx);
    return b < cross || (b == cross && __float_as_uint(e) >= e_min) ? e : 0.f;
  }
  return __float_as_uint(e) >= e_min ? e : 0.f;
}
__device__ __noinline__ float kept_mass_slow(float x, float mx, int cross, uint32_t e_min, uint32_t key_k) {
  return kept_mass_of(x, mx, cross, e_min, key_k);
}

// First bin at which the running sum over the bins (counts, or masses) reaches `target`, and the sum before it; the
// last bin when the target is never reached.  All threads call.
template <int NT, bool MASS>
__device__ __forceinline__ void find_crossing(Scratch* sc, double target, double lo_unit, double hi_unit) {
  constexpr int PER = SAMPLE_BINS / NT;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double v[PER], mine = 0.0;
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int b = tid * PER + j;
    v[j] = MASS ? (double)sc->bins[2][b] * hi_unit + (double)sc->bins[1][b] * lo_unit : (double)sc->bins[0][b];
    mine += v[j];
  }
  double inc = mine;
  for (int o = 1; o < 32; o <<= 1) {
    const double t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  __syncthreads();
  if (lane == 31) sc->warp_d[warp] = inc;
  if (tid == 0) { sc->cross_bin = SAMPLE_BINS - 1; sc->cross_before = 0.0; }
  __syncthreads();
  double before = inc - mine;
  for (int w = 0; w < warp; ++w) before += sc->warp_d[w];
  if ((before < target && target <= before + mine) || tid == NT - 1) {
    // (the last thread also covers a target that rounding put above the total)
    double cum = before;
    int b = 0;
#pragma unroll
    for (; b < PER - 1; ++b) {
      if (cum + v[b] >= target) break;
      cum += v[b];
    }
    if (before < target) { sc->cross_bin = tid * PER + b; sc->cross_before = cum; }
  }
  __syncthreads();
}

template <typename T, int NT>
__global__ void __launch_bounds__(NT, NT == 512 ? 2 : 1) k_sample_rows(SampleParams p) {
  extern __shared__ __align__(16) unsigned char dyn_smem[];
  __shared__ __align__(16) Scratch scratch;
  Scratch* sc = &scratch;
  const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  pdl_wait();
  pdl_trigger();

  int hrow = -1;
  if (p.history) {
    hrow = p.slot_ids ? p.slot_ids[row] : row;
    if (hrow < 0 || hrow >= p.n_hist_rows) hrow = -1;
  }
  if (p.slot_ids && hrow < 0 && p.history) {  // padded row of a captured batch: nothing to draw
    if (tid == 0) p.next_ids[row] = 0;
    return;
  }
  Row<T> r;
  r.init(reinterpret_cast<const T*>(p.logits) + (size_t)row * p.ldl, p.V);
  r.flat = p.inv_temperature == 0.f;
  r.inv_t = r.flat ? 1.f : p.inv_temperature;
  r.penalty = p.penalty;
  r.bits = nullptr;
  // the first loads of the row are on their way while the penalty's bits are set
  constexpr int VEC = Row<T>::VEC;
  const int per = (r.groups + NT / 32 - 1) / (NT / 32);
  const int g0 = warp * per, g1 = min(r.groups, (warp + 1) * per);      // this warp's stretch
  uint4 ahead[4];
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (g0 + lane + 32 * k < g1) ahead[k] = r.raw(g0 + lane + 32 * k);
  if (hrow >= 0 && p.penalty != 1.0f) {
    uint32_t* bm = p.bitmaps ? p.bitmaps + (size_t)row * p.bitmap_words : reinterpret_cast<uint32_t*>(dyn_smem);
    for (int i = tid; i < p.bitmap_words; i += NT) bm[i] = 0u;
    __syncthreads();
    int hlen = p.hist_len ? p.hist_len[hrow] : p.hist_cols;
    hlen = max(0, min(hlen, p.hist_cols));
    const int64_t* hist = p.history + (size_t)hrow * p.ld_hist;
    for (int j = tid; j < hlen; j += NT) {
      const int64_t h = hist[j];
      if (h >= 0 && h < p.V) atomicOr(&bm[((int)h + r.lead) >> 5], 1u << (((int)h + r.lead) & 31));
    }
    r.bits = bm;
  }
  if (tid == 0) { sc->n_list = sc->n_item = 0; sc->chosen = 0x7fffffff; sc->last_kept = -1; }
  __syncthreads();

  const bool use_k = p.top_k > 0 && p.top_k < p.V;
  const bool use_p = p.top_p > 0.f && p.top_p < 1.f;
  // ---- pass 1: the maximum, every thread's own, and (small top-k) that of each of its blocks: `steps` groups, 32 apart
  const bool want_list = use_k && p.top_k <= SAMPLE_LIST_TOP_K;
  const int most = SAMPLE_BLOCKS / NT, lane_groups = (per + 31) / 32;
  const int steps = (lane_groups + 4 * most - 1) / (4 * most) * 4, n_blocks = (lane_groups + steps - 1) / steps;
  float mine = -INFINITY, marked = -INFINITY;
  for (int b = 0; b < n_blocks; ++b) {
    RawMax<T> best;
    for (int k0 = 0; k0 < steps; k0 += 4) {
      const int g = g0 + lane + 32 * (b * steps + k0);
      uint4 u[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {        // the next four are requested before these are looked at
        u[k] = ahead[k];
        if (g + 32 * (4 + k) < g1) ahead[k] = r.raw(g + 32 * (4 + k));
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (g + 32 * k < g1) best.add(r.plain(g + 32 * k, u[k]));
    }
    const float v = best.value() * r.inv_t;       // (rounding is monotone: the scaled maximum is the maximum of the scaled)
    if (want_list || use_p) sc->blocks.top[b * NT + tid] = v;
    mine = fmaxf(mine, v);
  }
  for_marked<NT>(r, [&](int, float x) { marked = fmaxf(marked, x); });
  mine = fmaxf(mine, marked);
  const float mx = block_max<NT>(mine, sc);

  const float u = p.uniforms[row];
  float kept_mass = 0.f, kept_count = 0.f, z = 0.f;
  int pick = 0;
  bool listed = false;

  if (want_list) {
    // k-th largest of the threads' maxima, to its leading 20 bits (rounded down: still a lower bound), by one warp
    const uint32_t my_key = order_key(mine);
    sc->key[tid] = my_key;
    __syncthreads();
    if (warp == 0) {
      uint32_t keys[NT / 32], found = 0;
#pragma unroll
      for (int c = 0; c < NT / 32; ++c) keys[c] = sc->key[c * 32 + lane];
      for (int b = 31; b >= 12; --b) {
        const uint32_t t = found | (1u << b);
        int n = 0;
#pragma unroll
        for (int c = 0; c < NT / 32; ++c) n += keys[c] >= t;
        if (__reduce_add_sync(0xffffffffu, n) >= p.top_k) found = t;
      }
      if (lane == 0) sc->limit = found;
    }
    __syncthreads();
    const uint32_t bound = sc->limit;
    const float floor_x = key_value(bound);
    const bool all = bound <= 0x007fffffu;           // fewer than k threads hold a finite value: every element is listed
    if (all) {
      for_each<NT, true>(r, [&](int i, float x) {
        if ((unsigned)i < (unsigned)r.V) list_add(sc, order_key(x), i);
      });
    } else {
      for (int b = 0; b < n_blocks; ++b)
        if (sc->blocks.top[b * NT + tid] >= floor_x) {
          const int at = atomicAdd(&sc->n_item, 1);
          if (at < SAMPLE_ITEMS) sc->blocks.item[at] = b * NT + tid;
        }
      if (marked >= floor_x)
        for_marked<NT>(r, [&](int i, float x) {
          if (x >= floor_x) list_add(sc, order_key(x), i);
        });
      __syncthreads();
      const int n_item = min(sc->n_item, SAMPLE_ITEMS);
      for (int e = tid; e < n_item * steps; e += NT) {      // a group of a block for each thread
        const int it = sc->blocks.item[e / steps], b = it / NT, t = it - b * NT, w = t >> 5;
        const int g = w * per + (t & 31) + 32 * (b * steps + e % steps);
        if (g < min(r.groups, (w + 1) * per)) {
          float x[VEC];
          r.scaled(r.plain(g, r.raw(g)), x);
#pragma unroll
          for (int j = 0; j < VEC; ++j)
            if (x[j] >= floor_x) list_add(sc, order_key(x[j]), g * VEC - r.lead + j);
        }
      }
    }
    __syncthreads();
    const int m = sc->n_item > SAMPLE_ITEMS ? SAMPLE_LIST + 1 : sc->n_list;
    listed = m <= SAMPLE_LIST;                             // block-uniform
    if (listed) {
      const int m4 = (m + 3) & ~3;
      for (int j = m + tid; j < m4; j += NT) { sc->key[j] = 0u; sc->idx[j] = 0x7fffffff; }
      __syncthreads();
      // the k largest (ties with the k-th stay): fewer than k values above
      uint32_t kk[SAMPLE_LIST / NT];
#pragma unroll
      for (int c = 0; c < SAMPLE_LIST / NT; ++c) {
        const int j = tid + c * NT;
        kk[c] = 0u;
        if (j < m) {
          const uint32_t key = sc->key[j];
          int above = 0;
          for (int i = 0; i < m4; i += 4) {
            const uint4 o = *reinterpret_cast<const uint4*>(&sc->key[i]);
            above += (o.x > key) + (o.y > key) + (o.z > key) + (o.w > key);
          }
          if (above < p.top_k && mass_of(key_value(key), mx) > 0.f) kk[c] = key;
        }
      }
      __syncthreads();
#pragma unroll
      for (int c = 0; c < SAMPLE_LIST / NT; ++c)
        if (tid + c * NT < m) sc->key[tid + c * NT] = kk[c];
      __syncthreads();
      // vocabulary order: position = kept values with a smaller index
      int n_keep = 0;
#pragma unroll
      for (int c = 0; c < SAMPLE_LIST / NT; ++c) {
        const int j = tid + c * NT;
        if (kk[c]) {
          const int idx = sc->idx[j];
          int before = 0;
          for (int i = 0; i < m4; i += 4) {
            const uint4 o = *reinterpret_cast<const uint4*>(&sc->key[i]);
            const int4 q = *reinterpret_cast<const int4*>(&sc->idx[i]);
            before += (o.x && q.x < idx) + (o.y && q.y < idx) + (o.z && q.z < idx) + (o.w && q.w < idx);
          }
          sc->sorted.e[before] = mass_of(key_value(kk[c]), mx);
          sc->sorted.idx[before] = idx;
        }
      }
#pragma unroll
      for (int c = 0; c < SAMPLE_LIST / NT; ++c) n_keep += __syncthreads_count(kk[c] != 0u);
      // nucleus: keep a value when the mass above it is below top_p of the whole
      float e[SAMPLE_LIST / NT];
      if (tid < n_keep || tid == 0) {
        for (int i = 0; i < n_keep; ++i) z += sc->sorted.e[i];
      }
#pragma unroll
      for (int c = 0; c < SAMPLE_LIST / NT; ++c) {
        const int j = tid + c * NT;
        e[c] = 0.f;
        if (j < n_keep) {
          e[c] = sc->sorted.e[j];
          if (use_p) {
            float above = 0.f;
            for (int i = 0; i < n_keep; ++i) {
              const float o = sc->sorted.e[i];
              above += o > e[c] ? o : 0.f;
            }
            if (!(above < p.top_p * z)) e[c] = 0.f;
          }
        }
      }
      __syncthreads();
#pragma unroll
      for (int c = 0; c < SAMPLE_LIST / NT; ++c)
        if (tid + c * NT < n_keep) sc->sorted.e[tid + c * NT] = e[c];
      __syncthreads();
      // inverse CDF
#pragma unroll
      for (int c = 0; c < SAMPLE_LIST / NT; ++c) {
        const int j = tid + c * NT;
        if (e[c] > 0.f || j == 0) {
          float cum = 0.f, upto = 0.f, cnt = 0.f;
          for (int i = 0; i < n_keep; ++i) {
            const float o = sc->sorted.e[i];
            cum += o;
            cnt += o > 0.f ? 1.f : 0.f;
            if (i == j) upto = cum;
          }
          kept_mass = cum;
          kept_count = cnt;
          if (e[c] > 0.f) {
            atomicMax(&sc->last_kept, j);
            if (upto > u * cum) atomicMin(&sc->chosen, j);
          }
        }
      }
      __syncthreads();
      if (tid == 0) {
        const int at = sc->chosen != 0x7fffffff ? sc->chosen : sc->last_kept;
        pick = at >= 0 ? sc->sorted.idx[at] : 0;
      }
    }
  }

  if (!listed) {
    uint32_t key_k = 0u;                     // top-k: keep keys >= key_k
    int cross = SAMPLE_BINS;                 // top-p: keep bins < cross, and in bin `cross` the masses >= e_min
    uint32_t e_min = 1u;                     //        (cross == SAMPLE_BINS: e_min alone decides)
    float bin_lo = -INFINITY, bin_hi = INFINITY;      // below / above: the bin is certainly a later / an earlier one
    float all_mass = 0.f;
    if (use_k) {
      for (int b = tid; b < SAMPLE_BINS; b += NT) sc->bins[0][b] = 0u;
      if (tid == 0) sc->n_list = 0;
      __syncthreads();
      for_each<NT, true>(r, [&](int i, float x) {
        if ((unsigned)i < (unsigned)r.V) atomicAdd(&sc->bins[0][bin_of(x, mx)], 1u);
      });
      __syncthreads();
      find_crossing<NT, false>(sc, (double)p.top_k, 0.0, 0.0);
      const int cb = sc->cross_bin;
      const int need = p.top_k - (int)sc->cross_before;      // values to keep inside the bin
      for_each<NT, true>(r, [&](int i, float x) {
        if ((unsigned)i < (unsigned)r.V && bin_of(x, mx) == cb) list_add(sc, order_key(x), i);
      });
      if (tid == 0) sc->limit = 0xffffffffu;
      __syncthreads();
      const int m = sc->n_list;
      if (m <= SAMPLE_LIST) {
        for (int j = tid; j < m; j += NT) {
          const uint32_t key = sc->key[j];
          int above = 0;
          for (int i = 0; i < m; ++i) above += sc->key[i] > key;
          if (above < need) atomicMin(&sc->limit, key);
        }
        __syncthreads();
        key_k = sc->limit;
      } else {                               // a bin with more values than the list holds (mass ties): search the key's bits
        for (int b = 31; b >= 0; --b) {
          const uint32_t t = key_k | (1u << b);
          double c = 0.0;
          for_each<NT, true>(r, [&](int i, float x) {
            if ((unsigned)i < (unsigned)r.V && order_key(x) >= t) c += 1.0;
          });
          if (block_sum<NT>(c, sc) >= (double)p.top_k) key_k = t;
        }
      }
    }
    if (use_p) {
      const uint32_t half_mask = (1u << p.mass_half) - 1u;
      const float one = (float)(1u << (2 * p.mass_half));            // the integer that stands for e = 1
      const double unit = 1.0 / (double)one;
      // Values whose integer is at most `least` need no bin: all V of them together weigh less than (1 - top_p) of the
      // largest values of the blocks alone, so the nucleus closes before the first of them (and every bin in front of the one
      // it closes in is complete).  Two thirds of a row of 50 k normal logits.
      uint32_t least = 0u;
      if (!use_k) {
        unsigned long long some = 0ull;
        for (int b = 0; b < n_blocks; ++b) some += __float2uint_rn(mass_term(sc->blocks.top[b * NT + tid], mx) * one);
        const double share = (1.0 - (double)p.top_p) * block_sum<NT>((double)some, sc) / (double)p.V;
        if (share >= 2.0) least = (uint32_t)fmin(share, 1e9) - 1u;
      }
      for (int b = tid; b < SAMPLE_BINS; b += NT) sc->bins[1][b] = sc->bins[2][b] = 0u;
      __syncthreads();
      if (tid == 0) sc->n_list = 0;
      unsigned long long zz = 0ull;
      auto add_mass = [&](float x) {
        const float e = !use_k || order_key(x) >= key_k ? mass_term(x, mx) : 0.f;
        const uint32_t q = __float2uint_rn(e * one);
        zz += q;
        all_mass += e;
        if (q > least) {
          const int b = bin_of(x, mx);
          atomicAdd(&sc->bins[1][b], q & half_mask);
          if (q > half_mask) atomicAdd(&sc->bins[2][b], q >> p.mass_half);
        }
      };
      for_each<NT, false>(r, [&](int, float x) { add_mass(x); });
      for_marked<NT>(r, [&](int, float x) { add_mass(x); });
      const double zq = block_sum<NT>((double)zz, sc) * unit;     // exact: integers below 2^53
      const double target = (double)p.top_p * zq;
      find_crossing<NT, true>(sc, target, unit, unit * (double)(half_mask + 1u));
      cross = sc->cross_bin;
      const double before = sc->cross_before;
      // rough edges of the bin, wider than it by more than the rounding of mx - x and of the edges themselves (2^-23 of either)
      const float slack = 1e-6f * (fabsf(mx) + 33.f);
      if (cross > 0) bin_hi = mx - (float)cross * (1.f / SAMPLE_BINS_PER_UNIT) + slack;
      if (cross < SAMPLE_BINS - 1) bin_lo = mx - (float)(cross + 1) * (1.f / SAMPLE_BINS_PER_UNIT) - slack;
      auto add_bin = [&](int i, float x) {
        if (x >= bin_lo && x <= bin_hi) list_bin_value(sc, x, mx, i, cross, key_k);
      };
      for_each<NT, false>(r, add_bin);
      for_marked<NT>(r, add_bin);
      if (tid == 0) sc->limit = 0xffffffffu;
      __syncthreads();
      const int m = sc->n_list;
      if (m <= SAMPLE_LIST) {
        for (int j = tid; j < m; j += NT) {
          const uint32_t eb = sc->key[j];
          unsigned long long above = 0ull;
          for (int i = 0; i < m; ++i) {
            const uint32_t o = sc->key[i];
            if (o > eb) above += __float2uint_rn(__uint_as_float(o) * one);
          }
          if (before + (double)above * unit < target) atomicMin(&sc->limit, eb);
        }
        __syncthreads();
        e_min = sc->limit;
      } else {                               // mass ties: search the bits of the probability
        cross = SAMPLE_BINS;
        e_min = 0u;
        for (int b = 29; b >= 0; --b) {
          const uint32_t t = e_min | (1u << b);
          double c = 0.0;
          for_each<NT, true>(r, [&](int, float x) {
            const float e = order_key(x) >= key_k ? mass_of(x, mx) : 0.f;
            if (__float_as_uint(e) >= t) c += (double)__float2uint_rn(e * one);
          });
          if (block_sum<NT>(c, sc) * unit >= target) e_min = t;
        }
        e_min = max(e_min, 1u);
      }
    }
    auto keep = [&](float x) { return kept_mass_of(x, mx, cross, e_min, key_k); };
    // ---- masses of the warps' stretches (vocabulary order), then the stretch that holds the target is walked again
    float acc = 0.f;
    int cnt = 0;
    auto add_up = [&](auto kept) {
      auto add = [&](int, float x) {
        const float e = kept(x);
        acc += e;
        cnt += e > 0.f;
      };
      for_each<NT, false>(r, add);
      for_marked<NT>(r, add);
    };
    if (!use_k && !use_p) add_up([&](float x) { return mass_of(x, mx); });
    else if (!use_k)
      add_up([&](float x) {
        const float e = mass_term(x, mx);      // (where it is returned, above the bins' edge, it is at least e^-33)
        return x < bin_lo ? 0.f : x > bin_hi ? e : kept_mass_slow(x, mx, cross, e_min, 0u);
      });
    else add_up(keep);
    for (int o = 16; o; o >>= 1) {
      acc += __shfl_xor_sync(0xffffffffu, acc, o);
      cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    }
    __syncthreads();
    if (lane == 0) { sc->warp_f[warp] = acc; sc->warp_i[warp] = cnt; }
    __syncthreads();
    int total_cnt = 0, own = -1, last = -1;
    for (int w = 0; w < NT / 32; ++w) { kept_mass += sc->warp_f[w]; total_cnt += sc->warp_i[w]; }
    kept_count = (float)total_cnt;
    const float target = u * kept_mass;
    float before = 0.f, cum = 0.f;
    for (int w = 0; w < NT / 32; ++w) {
      if (sc->warp_i[w]) {
        last = w;
        if (own < 0 && cum + sc->warp_f[w] > target) { own = w; before = cum; }
      }
      cum += sc->warp_f[w];
    }
    const bool past_end = own < 0;           // u * total rounded up to the total: the last kept token
    if (past_end) own = last;
    z = use_p ? (float)block_sum<NT>((double)all_mass, sc) : kept_mass;
    // the stretch that holds the target, by the whole CTA: 16-byte groups in order, a running sum over them, then inside a group
    const int w0 = max(own, 0) * per, w1 = own < 0 ? 0 : min(r.groups, w0 + per);
    int last_i = -1;
    for (int base = w0; base < w1; base += NT) {      // (one round up to 50 k bf16 values)
      const int g = base + tid;
      float x[VEC], e[VEC], s = 0.f;
      if (g < w1) r.values(g, r.raw(g), x);
#pragma unroll
      for (int j = 0; j < VEC; ++j) {
        e[j] = g < w1 ? keep(x[j]) : 0.f;
        s += e[j];
        if (e[j] > 0.f) last_i = g * VEC - r.lead + j;
      }
      float inc = s;
      for (int o = 1; o < 32; o <<= 1) {
        const float t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
      }
      __syncthreads();
      if (lane == 31) sc->warp_f[warp] = inc;
      __syncthreads();
      float c = before, round = 0.f;
      for (int w = 0; w < NT / 32; ++w) {
        if (w == warp) c += round;
        round += sc->warp_f[w];
      }
      c += inc - s;
      before += round;
      if (!past_end) {
        int found = 0x7fffffff;
#pragma unroll
        for (int j = VEC - 1; j >= 0; --j) {
          float upto = c;
#pragma unroll
          for (int i = 0; i <= j; ++i) upto += e[i];
          if (e[j] > 0.f && upto > target) found = g * VEC - r.lead + j;
        }
        if (found != 0x7fffffff) atomicMin(&sc->chosen, found);
      }
    }
    if (last_i >= 0) atomicMax(&sc->last_kept, last_i);
    __syncthreads();
    if (tid == 0 && sc->chosen == 0x7fffffff) sc->chosen = sc->last_kept;
    __syncthreads();
    pick = sc->chosen;
    if (pick < 0 || pick >= p.V) pick = 0;
  }

  if (tid == 0) {
    p.next_ids[row] = pick;
    if (p.stats) {
      float* s = p.stats + 4 * (size_t)row;
      s[0] = mx;
      s[1] = kept_mass;
      s[2] = kept_count;
      s[3] = z;
    }
    if (p.append && hrow >= 0 && p.hist_len) {
      const int len = p.hist_len[hrow];
      if (len >= 0 && len < p.hist_cols) {
        p.history[(size_t)hrow * p.ld_hist + len] = pick;
        p.hist_len[hrow] = len + 1;
      }
    }
  }
}

template <typename T, int NT>
int sample_launch(const SampleParams& p, size_t smem, cudaStream_t st) {
  // the opt-in only ever grows (another thread may be between its opt-in and its launch for a larger vocabulary); allow_smem
  // reckons with 16 KB of static shared memory
  static_assert(sizeof(Scratch) >= 16 * 1024, "");
  const int rc = allow_smem(reinterpret_cast<const void*>(k_sample_rows<T, NT>), smem + sizeof(Scratch) - 16 * 1024);
  if (rc) return rc;
  launch_after(k_sample_rows<T, NT>, p.n, NT, smem, st, p);
  QPAM_LAUNCH_CHECK("k_sample_rows");
  return QPAM_OK;
}

}  // namespace
}  // namespace qpam

using namespace qpam;

extern "C" size_t qpam_sample_workspace_bytes(int32_t n, int32_t V) {
  if (n <= 0 || V <= 0) return 0;
  const size_t words = ((size_t)V + 8 + 31) / 32;
  return words * 4 <= SAMPLE_SMEM_BITMAP ? 0 : (size_t)n * words * 4;      // one bit per token, only for vocabularies beyond 1.3 M
}

extern "C" int qpam_sample_logits(const void* logits, int32_t io_dtype, int32_t n, int32_t V, int64_t ld_logits,
                                  float temperature, int32_t top_k, float top_p, float repetition_penalty,
                                  const int32_t* slot_ids, int64_t* history, int32_t n_hist_rows, int32_t hist_cols,
                                  int64_t ld_hist, int32_t* hist_len, int32_t append, const float* uniforms,
                                  int64_t* next_ids, float* stats, void* workspace, size_t workspace_bytes,
                                  void* stream) {
  QPAM_REQUIRE(logits && uniforms && next_ids, "sample: NULL pointer argument");
  QPAM_REQUIRE(io_dtype == QPAM_F32 || io_dtype == QPAM_BF16, "sample: io_dtype %d unknown", io_dtype);
  QPAM_REQUIRE(n >= 0 && V >= 1 && ld_logits >= V, "sample: bad n=%d V=%d ld=%lld", n, V, (long long)ld_logits);
  QPAM_REQUIRE(temperature > 0.f, "sample: temperature must be positive (arg-max decoding is qpam_head_argmax)");
  QPAM_REQUIRE(repetition_penalty > 0.f, "sample: repetition_penalty must be positive");
  QPAM_REQUIRE(top_k >= 0 && top_p >= 0.f, "sample: top_k and top_p must not be negative");
  QPAM_REQUIRE(!history || (n_hist_rows >= 1 && hist_cols >= 0 && ld_hist >= hist_cols), "sample: bad history shape");
  QPAM_REQUIRE(!append || (history && hist_len), "sample: append needs history and hist_len");
  if (n == 0) return QPAM_OK;
  SampleParams p{};
  p.logits = logits; p.ldl = ld_logits; p.slot_ids = slot_ids; p.history = history; p.ld_hist = ld_hist;
  p.hist_len = hist_len; p.uniforms = uniforms; p.next_ids = next_ids; p.stats = stats;
  p.n = n; p.V = V; p.n_hist_rows = n_hist_rows; p.hist_cols = hist_cols; p.top_k = top_k; p.append = append;
  p.inv_temperature = 1.f / temperature; p.top_p = top_p; p.penalty = repetition_penalty;
  const size_t need = qpam_sample_workspace_bytes(n, V);
  p.bitmap_words = (int)(((size_t)V + 8 + 31) / 32);
  p.mass_half = 15;
  while (p.mass_half > 1 && ((int64_t)V << p.mass_half) > (1ll << 32)) --p.mass_half;
  size_t smem = repetition_penalty != 1.f && history ? (size_t)p.bitmap_words * 4 : 0;
  if (need) {
    QPAM_REQUIRE(workspace && workspace_bytes >= need, "sample: workspace of %zu bytes needed, %zu given", need, workspace_bytes);
    p.bitmaps = reinterpret_cast<uint32_t*>(workspace);
    smem = 0;
  }
  // more rows than SMs: two CTAs of 512 threads share an SM, so that one row's block-wide steps run under the other's
  // passes; otherwise a row has an SM to itself and takes 1024 threads
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const bool wide = n <= sm_count();
  if (io_dtype == QPAM_F32) return wide ? sample_launch<float, 1024>(p, smem, st) : sample_launch<float, 512>(p, smem, st);
  return wide ? sample_launch<__nv_bfloat16, 1024>(p, smem, st) : sample_launch<__nv_bfloat16, 512>(p, smem, st);
}
