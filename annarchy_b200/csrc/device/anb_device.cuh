// Device-side building blocks shared by every generated network module.
//
// The generated source (annarchy_b200/generator/codegen.py) includes this
// text first, then declares one __constant__ pointer per device array
// (bound by the runtime) and the network's kernels, which call the
// templates below. Compiled by NVRTC for sm_100a.
//
// Numerics: the double-precision ("exact") kernels keep the reference's
// operation order — one sequential sum per row in ascending pre rank,
// conductance increments applied per post neuron in ascending pre rank —
// and the module is compiled without multiply-add contraction, so results
// are bit-identical to the reference CPU build compiled with
// -ffp-contract=off. The single-precision ("fast") kernels reorder sums
// freely (atomics, vector loads) and are checked against tolerances.
#pragma once

typedef unsigned int anb_u32;
typedef unsigned short anb_bf16;   // bfloat16 storage (upper half of an IEEE float)
typedef long long anb_i64;

#define ANB_WARP 32

// Error codes a kernel writes into the network's error word.
#ifndef M_PI
#define M_PI 3.14159265358979323846   // pi in equations (the reference's sympy output)
#endif
#define ANB_DEVERR_BARRIER_TIMEOUT 1
#define ANB_DEVERR_INDEX 2
#define ANB_DEVERR_MONITOR_OVERFLOW 3

// ---- built-in functions of the equation language --------------------------
// (names as emitted by the reference parser: ANNarchy/parser/ParserTemplate.py)
template <typename T> __device__ __forceinline__ T positive(T x) { return x > T(0) ? x : T(0); }
template <typename T> __device__ __forceinline__ T negative(T x) { return x < T(0) ? x : T(0); }
// modulo(a, b): the integer remainder of a and b truncated to 64-bit
// integers (the reference's `long(a) % long(b)`)
template <typename A, typename B>
__device__ __forceinline__ long long modulo(A a, B b) { return (long long)a % (long long)b; }
// power(x, a): x multiplied by itself, a converted to an unsigned integer
// exponent (the reference's integer power, a - 1 multiplications in order);
// an exponent of 0 gives x
__device__ __forceinline__ double power(double x, unsigned int a) {
  double r = x;
  for (unsigned int i = 1; i < a; ++i) r *= x;
  return r;
}
__device__ __forceinline__ float power(float x, unsigned int a) {
  float r = x;
  for (unsigned int i = 1; i < a; ++i) r *= x;
  return r;
}
__device__ __forceinline__ double power(int x, unsigned int a) { return power((double)x, a); }
#define clip(x, a, b) ((x) < (a) ? (a) : ((x) > (b) ? (b) : (x)))
#define ite(a, b, c) ((a) ? (b) : (c))

// ---- bfloat16 ---------------------------------------------------------------
__device__ __forceinline__ float anb_bf16_to_f32(anb_bf16 h) {
  return __uint_as_float(((anb_u32)h) << 16);
}
// Weight value in arithmetic precision: doubles stay double, floats float,
// bfloat16 is widened to float.
__device__ __forceinline__ double anb_wf(double w) { return w; }
__device__ __forceinline__ float anb_wf(float w) { return w; }
__device__ __forceinline__ float anb_wf(anb_bf16 w) { return anb_bf16_to_f32(w); }

// Rate r of neuron k of copy b, rounded to bfloat16 (nearest even), into the
// 64-neuron tiles of the batched block product: element (b, k % 64) of tile
// k / 64 in 8 x 8 core matrices of 16-byte rows.
__device__ __forceinline__ void anb_store_tile(anb_bf16* tiles, int b, int k, int copies, float r) {
  const anb_u32 u = __float_as_uint(r);
  tiles[(size_t)(k >> 6) * copies * 64 + ((b >> 3) * 8 + ((k & 63) >> 3)) * 64 + (b & 7) * 8 + (k & 7)] =
      (anb_bf16)((u + 0x7FFFu + ((u >> 16) & 1u)) >> 16);
}

// ---- spike bitmaps -------------------------------------------------------------
__device__ __forceinline__ bool anb_bit(const anb_u32* bits, int i) {
  return (bits[i >> 5] >> (i & 31)) & 1u;
}

// Start of every kernel of the grid engine's plan, which may be launched
// while the previous kernel of the stream still runs (programmatic dependent
// launch): wait until that kernel has finished and its writes are visible,
// then allow the next kernel to be scheduled. Outside such a launch both
// return at once.
__device__ __forceinline__ void anb_pdl_enter() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ void anb_report(int* err, int code) {
  if (err) atomicCAS(err, 0, code);
}

// ---- rate-coded weighted sums ------------------------------------------------------

// Thread per row, sequential sum in stored (ascending pre) order:
// sum[post_rank[row]] += sum_j w[j] * r[col[j]]  (double, reference order).
template <typename R, typename W, typename I>
__device__ __forceinline__ void anb_rate_csr_scalar(int n_rows, const I* __restrict__ row_ptr,
                                                    const int* __restrict__ col,
                                                    const W* __restrict__ w,
                                                    const R* __restrict__ pre_r,
                                                    const int* __restrict__ post_rank,
                                                    R* __restrict__ sum) {
  for (int row = blockIdx.x * blockDim.x + threadIdx.x; row < n_rows;
       row += gridDim.x * blockDim.x) {
    R s = R(0);
    const I beg = row_ptr[row], end = row_ptr[row + 1];
    for (I j = beg; j < end; ++j) s += pre_r[col[j]] * (R)w[j];
    const int post = post_rank ? post_rank[row] : row;
    sum[post] += s;
  }
}

// Warp per row, the same sum in the same order as anb_rate_csr_scalar: the
// lanes form 32 products pre_r[col[j]] * w[j] at a time (coalesced index and
// weight loads, all gathers in flight, the next 32 loading while these are
// added), then every lane adds them one by one in stored order, as the
// reference's sequential loop does (ANNarchy/generator/Projection/OpenMP/
// CSR.py:177-253); no addition is reordered, so the result is the scalar
// kernel's bit for bit.
template <typename R, typename W, typename I>
__device__ __forceinline__ void anb_rate_csr_ordered(int n_rows, const I* __restrict__ row_ptr,
                                                     const int* __restrict__ col,
                                                     const W* __restrict__ w,
                                                     const R* __restrict__ pre_r,
                                                     const int* __restrict__ post_rank,
                                                     R* __restrict__ sum) {
  const int lane = threadIdx.x & 31;
  const int nwarps = (int)((gridDim.x * blockDim.x) >> 5);
  for (int row = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); row < n_rows; row += nwarps) {
    const I beg = row_ptr[row], end = row_ptr[row + 1];
    R s = R(0);
    I j = beg + lane;
    R p = j < end ? pre_r[col[j]] * (R)w[j] : R(0);
    for (I j0 = beg; j0 < end; j0 += 32) {
      const I jn = j0 + 32 + lane;
      const R pn = jn < end ? pre_r[col[jn]] * (R)w[jn] : R(0);
      if (end - j0 >= 32) {
#pragma unroll
        for (int k = 0; k < 32; ++k) s += __shfl_sync(0xffffffffu, p, k);
      } else {
        const int cnt = (int)(end - j0);
        for (int k = 0; k < cnt; ++k) s += __shfl_sync(0xffffffffu, p, k);
      }
      p = pn;
    }
    if (lane == 0) sum[post_rank ? post_rank[row] : row] += s;
  }
}

// ---- random numbers in equations --------------------------------------------------------
// Counter-based generator Philox4x32-10 (J. K. Salmon, M. A. Moraes, R. O. Dror,
// D. E. Shaw, "Parallel random numbers: as easy as 1, 2, 3", SC'11): ten
// rounds of two 32x32->64 multiplications with the published multipliers
// and Weyl key increments. A draw is a pure function of (seed, stream,
// step, neuron), so no generator state is stored or advanced, and every
// neuron of every step draws independently in any launch order.
struct anb_u4 {
  unsigned x, y, z, w;
};

__device__ __forceinline__ anb_u4 anb_philox4x32_10(anb_u4 c, unsigned k0, unsigned k1) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const unsigned long long p0 = (unsigned long long)0xD2511F53u * c.x;
    const unsigned long long p1 = (unsigned long long)0xCD9E8D57u * c.z;
    const unsigned hi0 = (unsigned)(p0 >> 32), lo0 = (unsigned)p0;
    const unsigned hi1 = (unsigned)(p1 >> 32), lo1 = (unsigned)p1;
    c = anb_u4{hi1 ^ c.y ^ k0, lo1, hi0 ^ c.w ^ k1, lo0};
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  return c;
}

// The four 32-bit words of draw (seed, stream, step t, index i).
__device__ __forceinline__ anb_u4 anb_rand_words(const unsigned* seed, unsigned stream, long long t,
                                                 unsigned i) {
  return anb_philox4x32_10(anb_u4{i, (unsigned)t, (unsigned)((unsigned long long)t >> 32), stream},
                           seed[0], seed[1]);
}

// Uniform on [0, 1): 24 bits (float) or 53 bits (double) of the first words.
template <typename R>
__device__ __forceinline__ R anb_unit(const anb_u4& w);
template <>
__device__ __forceinline__ float anb_unit<float>(const anb_u4& w) {
  return (float)(w.x >> 8) * (1.0f / 16777216.0f);
}
template <>
__device__ __forceinline__ double anb_unit<double>(const anb_u4& w) {
  return (double)(((unsigned long long)(w.x >> 6) << 27) | (w.y >> 5)) * (1.0 / 9007199254740992.0);
}

// Standard normal by the Box-Muller transform of two uniforms (the second
// pair of words); u1 in (0, 1] keeps the logarithm finite.
template <typename R>
__device__ __forceinline__ R anb_std_normal(const anb_u4& w) {
  const anb_u4 v{w.z, w.w, w.x, w.y};
  const R u1 = R(1) - anb_unit<R>(w), u2 = anb_unit<R>(v);
  return sqrt(R(-2) * log(u1)) * cos(R(6.283185307179586) * u2);
}

template <typename R>
__device__ __forceinline__ R anb_draw_uniform(const unsigned* seed, unsigned stream, long long t,
                                              unsigned i, R lo, R hi) {
  return lo + (hi - lo) * anb_unit<R>(anb_rand_words(seed, stream, t, i));
}
template <typename R>
__device__ __forceinline__ R anb_draw_normal(const unsigned* seed, unsigned stream, long long t,
                                             unsigned i, R mu, R sigma) {
  return mu + sigma * anb_std_normal<R>(anb_rand_words(seed, stream, t, i));
}
template <typename R>
__device__ __forceinline__ R anb_draw_lognormal(const unsigned* seed, unsigned stream, long long t,
                                                unsigned i, R mu, R sigma) {
  return exp(mu + sigma * anb_std_normal<R>(anb_rand_words(seed, stream, t, i)));
}
template <typename R>
__device__ __forceinline__ R anb_draw_exponential(const unsigned* seed, unsigned stream, long long t,
                                                  unsigned i, R lambda) {
  return -log(R(1) - anb_unit<R>(anb_rand_words(seed, stream, t, i))) / lambda;
}
template <typename R>
__device__ __forceinline__ R anb_draw_discrete_uniform(const unsigned* seed, unsigned stream, long long t,
                                                       unsigned i, R lo, R hi) {
  return lo + floor(anb_unit<R>(anb_rand_words(seed, stream, t, i)) * (hi - lo + R(1)));
}

// Slot of time step s (possibly negative) in a ring of `slots` entries.
__device__ __forceinline__ int anb_ring_slot(long long s, int slots) {
  const long long m = s % slots;
  return (int)(m < 0 ? m + slots : m);
}

// Rate-coded weighted sum with one transmission delay per synapse (steps,
// >= 1): thread per row, sequential in stored order like anb_rate_csr_scalar,
// each rate read from the pre population's history ring (slot of step
// t - delay; slots x n_pre values). The reference's non-uniform delays read
// pre.r from its queue entry delay - 1 (ANNarchy/generator/Projection/
// SingleThreadGenerator.py, _computesum_rate with max_delay > 1).
// The same sum with a warp per row (products gathered 32 at a time, added
// one by one in stored order, as anb_rate_csr_ordered).
template <typename R, typename W, typename I>
__device__ __forceinline__ void anb_rate_csr_delayed_ordered(int n_rows, const I* __restrict__ row_ptr,
                                                             const int* __restrict__ col,
                                                             const W* __restrict__ w,
                                                             const int* __restrict__ dly,
                                                             const R* __restrict__ ring, int n_pre,
                                                             int slots, long long t,
                                                             const int* __restrict__ post_rank,
                                                             R* __restrict__ sum) {
  const int lane = threadIdx.x & 31;
  const int nwarps = (int)((gridDim.x * blockDim.x) >> 5);
  for (int row = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); row < n_rows; row += nwarps) {
    const I beg = row_ptr[row], end = row_ptr[row + 1];
    R s = R(0);
    I j = beg + lane;
    R p = j < end ? ring[(size_t)anb_ring_slot(t - dly[j], slots) * n_pre + col[j]] * (R)w[j] : R(0);
    for (I j0 = beg; j0 < end; j0 += 32) {
      const I jn = j0 + 32 + lane;
      const R pn = jn < end ? ring[(size_t)anb_ring_slot(t - dly[jn], slots) * n_pre + col[jn]] * (R)w[jn]
                            : R(0);
      const int cnt = end - j0 >= 32 ? 32 : (int)(end - j0);
      for (int k = 0; k < cnt; ++k) s += __shfl_sync(0xffffffffu, p, k);
      p = pn;
    }
    if (lane == 0) sum[post_rank ? post_rank[row] : row] += s;
  }
}

template <typename R, typename W, typename I>
__device__ __forceinline__ void anb_rate_csr_delayed(int n_rows, const I* __restrict__ row_ptr,
                                                     const int* __restrict__ col,
                                                     const W* __restrict__ w,
                                                     const int* __restrict__ dly,
                                                     const R* __restrict__ ring, int n_pre,
                                                     int slots, long long t,
                                                     const int* __restrict__ post_rank,
                                                     R* __restrict__ sum) {
  for (int row = blockIdx.x * blockDim.x + threadIdx.x; row < n_rows;
       row += gridDim.x * blockDim.x) {
    R s = R(0);
    const I beg = row_ptr[row], end = row_ptr[row + 1];
    for (I j = beg; j < end; ++j)
      s += ring[(size_t)anb_ring_slot(t - dly[j], slots) * n_pre + col[j]] * (R)w[j];
    const int post = post_rank ? post_rank[row] : row;
    sum[post] += s;
  }
}

// Sub-warp per row (G lanes, G in {2,4,8,16,32}), fp32 accumulation with a
// butterfly reduction. Rows longer than `kahan_min` use compensated
// (Kahan) summation per lane.
template <int G, typename W, typename I>
__device__ __forceinline__ void anb_rate_csr_vector(int n_rows, const I* __restrict__ row_ptr,
                                                    const int* __restrict__ col,
                                                    const W* __restrict__ w,
                                                    const float* __restrict__ pre_r,
                                                    const int* __restrict__ post_rank,
                                                    float* __restrict__ sum, int kahan_min) {
  const int lane = threadIdx.x % G;
  const int groups = (gridDim.x * blockDim.x) / G;
  for (int row = (blockIdx.x * blockDim.x + threadIdx.x) / G; row < n_rows; row += groups) {
    const I beg = row_ptr[row], end = row_ptr[row + 1];
    float s = 0.f;
    if (end - beg >= (I)kahan_min) {
      float c = 0.f;
      for (I j = beg + lane; j < end; j += G) {
        float y = __fmul_rn(__ldg(&pre_r[__ldg(&col[j])]), anb_wf(w[j])) - c;
        float t = s + y;
        c = (t - s) - y;
        s = t;
      }
    } else {
      for (I j = beg + lane; j < end; j += G) s += __ldg(&pre_r[__ldg(&col[j])]) * anb_wf(w[j]);
    }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o, G);
    if (lane == 0) {
      const int post = post_rank ? post_rank[row] : row;
      sum[post] += s;
    }
  }
}

// Streaming loads of matrix data that is read once per step: not allocated
// in L1, so L1 keeps the gathered pre-synaptic vector.
__device__ __forceinline__ int4 anb_ls_i4(const int4* p) {
  int4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.s32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ float4 anb_ls_f4(const float4* p) {
  float4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint2 anb_ls_u2(const uint2* p) {
  uint2 v;
  asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ int anb_ls_i(const int* p) {
  int v;
  asm volatile("ld.global.nc.L1::no_allocate.s32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float anb_ls_f(const float* p) {
  float v;
  asm volatile("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ unsigned short anb_ls_h(const unsigned short* p) {
  unsigned short v;
  asm volatile("ld.global.nc.L1::no_allocate.u16 %0, [%1];" : "=h"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ uint4 anb_ls_u4(const uint4* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ anb_u32 anb_ls_u(const anb_u32* p) {
  anb_u32 v;
  asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// Bulk prefetch of a byte range of global memory into L2; the address and
// the size are multiples of 16 bytes and the range lies inside one array.
__device__ __forceinline__ void anb_prefetch_l2(const void* p, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" :: "l"(p), "r"(bytes) : "memory");
}

// Four consecutive weights widened to float (16-byte or 8-byte load).
__device__ __forceinline__ float4 anb_w4(const float* w) { return anb_ls_f4(reinterpret_cast<const float4*>(w)); }
__device__ __forceinline__ float4 anb_w4(const anb_bf16* w) {
  const uint2 u = anb_ls_u2(reinterpret_cast<const uint2*>(w));
  return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u),
                     __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
}
__device__ __forceinline__ float anb_w1(const float* w) { return anb_ls_f(w); }
__device__ __forceinline__ float anb_w1(const anb_bf16* w) { return anb_bf16_to_f32(anb_ls_h(w)); }

// Sub-warp per row with 16-byte vector loads of the column indices and
// weights (streaming, evict-first) over the 4-aligned body of every row and
// scalar loads at its ends. `rows` (optional) lists the rows to process
// (row-length binning); `n_rows` is its length. SET: nothing else is added to
// these sums (a store does not wait for the old value).
template <int G, typename W, bool SET = false>
__device__ __forceinline__ void anb_rate_csr_vec(int n_rows, const int* __restrict__ rows,
                                                 const int* __restrict__ row_ptr,
                                                 const int* __restrict__ col,
                                                 const W* __restrict__ w,
                                                 const float* __restrict__ x,
                                                 const int* __restrict__ post_rank,
                                                 float* __restrict__ sum) {
  const int lane = threadIdx.x % G;
  const int groups = (gridDim.x * blockDim.x) / G;
  // (a warp's lanes stay together: all of them take part in the shuffles)
  const int in_warp = (threadIdx.x & 31) / G;
  for (int r = (blockIdx.x * blockDim.x + threadIdx.x) / G; r - in_warp < n_rows; r += groups) {
    const int row = r >= n_rows ? -1 : rows ? rows[r] : r;
    const int beg = row < 0 ? 0 : row_ptr[row], end = row < 0 ? 0 : row_ptr[row + 1];
    int j0 = (beg + 3) & ~3;
    if (j0 > end) j0 = end;
    float s = 0.f;
    for (int j = beg + lane; j < j0; j += G) s += __ldg(&x[anb_ls_i(&col[j])]) * anb_w1(&w[j]);
    const int nv = (end - j0) >> 2;
    const int4* __restrict__ c4 = reinterpret_cast<const int4*>(col + j0);
    float s1 = 0.f;
    int v = lane;
    for (; v + G < nv; v += 2 * G) {          // two vectors in flight per lane
      const int4 ca = anb_ls_i4(c4 + v), cb = anb_ls_i4(c4 + v + G);
      const float4 wa = anb_w4(w + j0 + 4 * v), wb = anb_w4(w + j0 + 4 * (v + G));
      s += __ldg(&x[ca.x]) * wa.x + __ldg(&x[ca.y]) * wa.y + __ldg(&x[ca.z]) * wa.z +
           __ldg(&x[ca.w]) * wa.w;
      s1 += __ldg(&x[cb.x]) * wb.x + __ldg(&x[cb.y]) * wb.y + __ldg(&x[cb.z]) * wb.z +
            __ldg(&x[cb.w]) * wb.w;
    }
    if (v < nv) {
      const int4 c = anb_ls_i4(c4 + v);
      const float4 ww = anb_w4(w + j0 + 4 * v);
      s += __ldg(&x[c.x]) * ww.x + __ldg(&x[c.y]) * ww.y + __ldg(&x[c.z]) * ww.z +
           __ldg(&x[c.w]) * ww.w;
    }
    s += s1;
    for (int j = j0 + 4 * nv + lane; j < end; j += G) s += __ldg(&x[anb_ls_i(&col[j])]) * anb_w1(&w[j]);
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o, G);
    if (lane == 0 && row >= 0) {
      float* const to = &sum[post_rank ? post_rank[row] : row];
      *to = SET ? s : *to + s;
    }
  }
}

// One CTA per (long) row, Kahan-compensated per thread, block reduction.
template <typename W>
__device__ __forceinline__ void anb_rate_csr_cta(int n_rows, const int* __restrict__ rows,
                                                 const int* __restrict__ row_ptr,
                                                 const int* __restrict__ col,
                                                 const W* __restrict__ w,
                                                 const float* __restrict__ x,
                                                 const int* __restrict__ post_rank,
                                                 float* __restrict__ sum) {
  __shared__ float red[32];
  for (int r = blockIdx.x; r < n_rows; r += gridDim.x) {
    const int row = rows ? rows[r] : r;
    const int beg = row_ptr[row], end = row_ptr[row + 1];
    float s = 0.f, c = 0.f;
    for (int j = beg + threadIdx.x; j < end; j += blockDim.x) {
      const float y = __fmul_rn(__ldg(&x[anb_ls_i(&col[j])]), anb_w1(&w[j])) - c;
      const float t = s + y;
      c = (t - s) - y;
      s = t;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
      float v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.f;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (threadIdx.x == 0) sum[post_rank ? post_rank[row] : row] += v;
    }
    __syncthreads();
  }
}

// Blocked CSR with T x T tiles stored column-major (val[tile][c][r]): one
// CTA per block row; thread (r, part) sums tile row r over its share of the
// tile columns, then the parts are added in shared memory. Exact mode keeps
// one part per row (ascending columns = ascending pre rank).
template <int T, int PARTS, typename R, typename W>
__device__ __forceinline__ void anb_rate_bsr_rows(int n_block_rows, const int* __restrict__ brow_ptr,
                                                  const int* __restrict__ bcol,
                                                  const W* __restrict__ val,
                                                  const R* __restrict__ x, int n_pre, int n_post,
                                                  R* __restrict__ sum) {
  __shared__ R part[PARTS][T];
  const int r = threadIdx.x % T, pidx = threadIdx.x / T;
  constexpr int CW = T / PARTS;
  for (int br = blockIdx.x; br < n_block_rows; br += gridDim.x) {
    R s = R(0);
    if (pidx < PARTS) {
      for (int b = brow_ptr[br]; b < brow_ptr[br + 1]; ++b) {
        const W* __restrict__ tile = val + (size_t)b * T * T;
        const int c0 = bcol[b] * T;
        const R* __restrict__ xs = x + c0;
        const int cend = min((pidx + 1) * CW, n_pre - c0);   // partial last tile column
        for (int c = pidx * CW; c < cend; ++c) s += xs[c] * (R)anb_wf(tile[c * T + r]);
      }
      part[pidx][r] = s;
    }
    __syncthreads();
    if (pidx == 0) {
      R tot = part[0][r];
      for (int q = 1; q < PARTS; ++q) tot += part[q][r];
      const int post = br * T + r;
      if (post < n_post) sum[post] += tot;
    }
    __syncthreads();
  }
}

// ELLPACK / ELLPACK-R: column-major slots, thread per row.
// cols[k*n_rows + row], w likewise; rl = row lengths (ELL-R) or nullptr
// (ELL: stop at the first slot holding -1).
template <typename R, typename W>
__device__ __forceinline__ void anb_rate_ell(int n_rows, int width, const int* __restrict__ cols,
                                             const W* __restrict__ w, const int* __restrict__ rl,
                                             const R* __restrict__ pre_r,
                                             const int* __restrict__ post_rank,
                                             R* __restrict__ sum) {
  for (int row = blockIdx.x * blockDim.x + threadIdx.x; row < n_rows;
       row += gridDim.x * blockDim.x) {
    const int len = rl ? rl[row] : width;
    R s = R(0);
    if (sizeof(R) == 8 || !rl) {
      // exact order (double) or ELL with -1 padding: one chain
      for (int k = 0; k < len; ++k) {
        const int c = cols[(size_t)k * n_rows + row];
        if (!rl && c < 0) break;
        s += pre_r[c] * (R)anb_wf(w[(size_t)k * n_rows + row]);
      }
    } else {
      // four independent chains keep four gathers in flight per thread
      R s1 = R(0), s2 = R(0), s3 = R(0);
      int k = 0;
      for (; k + 4 <= len; k += 4) {
        const size_t o = (size_t)k * n_rows + row;
        const int c0 = __ldcs(&cols[o]), c1 = __ldcs(&cols[o + n_rows]);
        const int c2 = __ldcs(&cols[o + 2 * (size_t)n_rows]), c3 = __ldcs(&cols[o + 3 * (size_t)n_rows]);
        const R w0 = (R)anb_wf(w[o]), w1 = (R)anb_wf(w[o + n_rows]);
        const R w2 = (R)anb_wf(w[o + 2 * (size_t)n_rows]), w3 = (R)anb_wf(w[o + 3 * (size_t)n_rows]);
        s += __ldg(&pre_r[c0]) * w0;
        s1 += __ldg(&pre_r[c1]) * w1;
        s2 += __ldg(&pre_r[c2]) * w2;
        s3 += __ldg(&pre_r[c3]) * w3;
      }
      for (; k < len; ++k) {
        const size_t o = (size_t)k * n_rows + row;
        s += __ldg(&pre_r[__ldcs(&cols[o])]) * (R)anb_wf(w[o]);
      }
      s = (s + s1) + (s2 + s3);
    }
    const int post = post_rank ? post_rank[row] : row;
    sum[post] += s;
  }
}

// ELL / ELL-R / SELL in single precision with G threads per row: a CTA of
// R*G threads covers R consecutive rows (consecutive lanes = consecutive rows,
// so every load instruction is one contiguous run); thread part g takes slots
// g, g+G, ...; the G partial sums are added in shared memory.
// SELL passes its slice layout (slot of (row, k) = slice_ptr[row/C] + k*C + row%C);
// ELL passes slice_ptr = nullptr (slot = k*n_rows + row).
template <int G, int C, typename W>
__device__ __forceinline__ void anb_rate_slots_split(int n_rows, int width,
                                                     const int* __restrict__ slice_ptr,
                                                     const int* __restrict__ cols,
                                                     const W* __restrict__ w,
                                                     const int* __restrict__ rl,
                                                     const int* __restrict__ perm,
                                                     const float* __restrict__ x,
                                                     const int* __restrict__ post_rank,
                                                     float* __restrict__ sum) {
  __shared__ float part[1024];
  const int R = blockDim.x / G;
  const int lr = threadIdx.x % R, g = threadIdx.x / R;
  for (int base = blockIdx.x * R; base < n_rows; base += gridDim.x * R) {
    const int r = base + lr;
    float s = 0.f, s1 = 0.f;
    if (r < n_rows) {
      const int len = rl ? rl[r] : width;
      size_t slot0, stride;
      if (slice_ptr) {
        slot0 = (size_t)slice_ptr[r / C] + (r % C);
        stride = C;
      } else {
        slot0 = r;
        stride = (size_t)n_rows;
      }
      int k = g;
      for (; k + G < len; k += 2 * G) {
        const size_t o0 = slot0 + (size_t)k * stride, o1 = o0 + (size_t)G * stride;
        const int c0 = anb_ls_i(&cols[o0]), c1 = anb_ls_i(&cols[o1]);
        if (!rl && c1 < 0) {
          if (c0 >= 0) s += __ldg(&x[c0]) * anb_w1(&w[o0]);
          k = len;
          break;
        }
        s += __ldg(&x[c0]) * anb_w1(&w[o0]);
        s1 += __ldg(&x[c1]) * anb_w1(&w[o1]);
      }
      if (k < len) {
        const size_t o0 = slot0 + (size_t)k * stride;
        const int c0 = anb_ls_i(&cols[o0]);
        if (rl || c0 >= 0) s += __ldg(&x[c0]) * anb_w1(&w[o0]);
      }
    }
    part[threadIdx.x] = s + s1;
    __syncthreads();
    if (g == 0 && r < n_rows) {
      float tot = part[lr];
      for (int q = 1; q < G; ++q) tot += part[lr + q * R];
      const int row = perm ? perm[r] : r;
      sum[post_rank ? post_rank[row] : row] += tot;
    }
    __syncthreads();
  }
}

// SELL-C-sigma: slices of C consecutive (sorted) rows, column-major inside
// a slice; slice_ptr[s] = first slot of slice s, slice_len[s] = its width.
// perm[row in slice order] = original row. Thread per row.
template <int C, typename R, typename W>
__device__ __forceinline__ void anb_rate_sell(int n_rows, const int* __restrict__ slice_ptr,
                                              const int* __restrict__ slice_len,
                                              const int* __restrict__ cols,
                                              const W* __restrict__ w,
                                              const int* __restrict__ row_len,
                                              const int* __restrict__ perm,
                                              const R* __restrict__ pre_r,
                                              const int* __restrict__ post_rank,
                                              R* __restrict__ sum) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n_rows; r += gridDim.x * blockDim.x) {
    const int sl = r / C, lane = r % C;
    const int base = slice_ptr[sl];
    const int len = row_len[r];
    R s = R(0);
    if (sizeof(R) == 8) {
      for (int k = 0; k < len; ++k) {
        const int slot = base + k * C + lane;
        s += pre_r[cols[slot]] * (R)anb_wf(w[slot]);
      }
    } else {
      R s1 = R(0), s2 = R(0), s3 = R(0);
      int k = 0;
      for (; k + 4 <= len; k += 4) {
        const int o = base + k * C + lane;
        const int c0 = __ldcs(&cols[o]), c1 = __ldcs(&cols[o + C]);
        const int c2 = __ldcs(&cols[o + 2 * C]), c3 = __ldcs(&cols[o + 3 * C]);
        const R w0 = (R)anb_wf(w[o]), w1 = (R)anb_wf(w[o + C]);
        const R w2 = (R)anb_wf(w[o + 2 * C]), w3 = (R)anb_wf(w[o + 3 * C]);
        s += __ldg(&pre_r[c0]) * w0;
        s1 += __ldg(&pre_r[c1]) * w1;
        s2 += __ldg(&pre_r[c2]) * w2;
        s3 += __ldg(&pre_r[c3]) * w3;
      }
      for (; k < len; ++k) {
        const int o = base + k * C + lane;
        s += __ldg(&pre_r[__ldcs(&cols[o])]) * (R)anb_wf(w[o]);
      }
      s = (s + s1) + (s2 + s3);
    }
    const int row = perm ? perm[r] : r;
    const int post = post_rank ? post_rank[row] : row;
    sum[post] += s;
  }
}

// COO tail of HYB: one thread per entry, atomic accumulation (fast mode) —
// the exact mode runs the tail with one thread per row instead.
template <typename W>
__device__ __forceinline__ void anb_rate_coo_atomic(int nnz, const int* __restrict__ rows,
                                                    const int* __restrict__ cols,
                                                    const W* __restrict__ w,
                                                    const float* __restrict__ pre_r,
                                                    const int* __restrict__ post_rank,
                                                    float* __restrict__ sum) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nnz; k += gridDim.x * blockDim.x) {
    const int row = rows[k];
    const int post = post_rank ? post_rank[row] : row;
    atomicAdd(&sum[post], pre_r[cols[k]] * anb_wf(w[k]));
  }
}

// ---- panelled sliced ELL (fast mode) ------------------------------------------------
// The pre-synaptic columns are cut into panels of at most `panel_width`
// neurons (16-bit column indices relative to the panel). Within a panel the
// rows are sorted by their number of synapses there and cut into slices of 32
// rows stored as steps of 32 elements, one per row: a header step naming the
// rows, then element k of every row at step k + 1. A CTA copies its panel's
// rates into shared memory with bulk (TMA) copies; each warp then streams a
// contiguous range of steps, one row per lane, loading the next chunk of U
// steps while it sums the current one, and adds its partial sum to the row's
// global sum where a slice (or its range) ends.

// Issue bulk copies of `bytes` (a multiple of 16, both addresses 16-byte
// aligned) from global memory into this CTA's shared memory, completing on
// the mbarrier `mbar` (phase 0). Called by one thread; the barrier must be
// published (CTA barrier) before other threads wait on it.
__device__ __forceinline__ void anb_bulk_issue(void* dst, const void* src, unsigned bytes,
                                               unsigned long long* mbar) {
  const unsigned mb = (unsigned)__cvta_generic_to_shared(mbar);
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("{ .reg .b64 st; mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1; }"
               ::"r"(mb), "r"(bytes) : "memory");
  const unsigned chunk = 32768u;
  for (unsigned off = 0; off < bytes; off += chunk) {
    const unsigned n = bytes - off < chunk ? bytes - off : chunk;
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
        ::"r"(d + off), "l"(reinterpret_cast<const char*>(src) + off), "r"(n), "r"(mb)
        : "memory");
  }
}

// Wait for phase 0 of `mbar`, at most ANB_BULK_WAIT_TRIES polls; a timeout is
// reported in `err` (the copied data is then incomplete; the kernel still
// finishes).
#define ANB_BULK_WAIT_TRIES (1 << 22)
__device__ __forceinline__ void anb_bulk_wait(unsigned long long* mbar, int* err) {
  const unsigned mb = (unsigned)__cvta_generic_to_shared(mbar);
  unsigned done = 0;
  for (int it = 0; it < ANB_BULK_WAIT_TRIES && !done; ++it) {
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0; selp.u32 %0, 1, 0, p; }"
        : "=r"(done) : "r"(mb) : "memory");
  }
  if (!done) anb_report(err, ANB_DEVERR_BARRIER_TIMEOUT);
}

// Eight consecutive weights (aligned) widened to float.
__device__ __forceinline__ void anb_w8(const float* w, float* o) {
  const float4 a = anb_ls_f4(reinterpret_cast<const float4*>(w));
  const float4 b = anb_ls_f4(reinterpret_cast<const float4*>(w) + 1);
  o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w; o[4] = b.x; o[5] = b.y; o[6] = b.z; o[7] = b.w;
}
__device__ __forceinline__ void anb_w8(const anb_bf16* w, float* o) {
  const uint4 u = anb_ls_u4(reinterpret_cast<const uint4*>(w));
  const anb_u32 q[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    o[2 * i] = __uint_as_float(q[i] << 16);
    o[2 * i + 1] = __uint_as_float(q[i] & 0xffff0000u);
  }
}

// Sum index of a header entry (column c, weight slot read as wv): the entry
// stores v = index + 1 (0 for a padding lane) as column 0xF000 | (v >> 16)
// and the weight slot's bits v (32-bit weights) or v & 0xffff (bfloat16).
__device__ __forceinline__ int anb_pc_row(unsigned c, float wv, const float*) {
  return __float_as_int(wv) - 1;
}
__device__ __forceinline__ int anb_pc_row(unsigned c, float wv, const anb_bf16*) {
  return (int)(((c & 0xfffu) << 16) | (__float_as_uint(wv) >> 16)) - 1;
}

// cta_panel[blockIdx.x]: the CTA's panel; warp_tab[3 * (blockIdx.x * warps
// + warp) ...] = (first step, end step, header step of the slice holding the
// first step); col / w: 32 entries per step, columns from 0xF000 on marking
// header steps. Dynamic shared memory: panel_width floats.
// Weight of a pcsr entry as float (streaming load; the compiler folds the
// constant step offsets of a chunk into the load addresses).
__device__ __forceinline__ float anb_pc_w(const float* w) { return __ldcs(w); }
__device__ __forceinline__ float anb_pc_w(const anb_bf16* w) {
  return __uint_as_float((unsigned)__ldcs(reinterpret_cast<const unsigned short*>(w)) << 16);
}

//
// wait(): called once, after what the step does not change (the work split and
// the first entries) has been asked for and before x is read.
template <typename W, int U, typename Wait>
__device__ __forceinline__ void anb_rate_pcsr(const int* __restrict__ cta_panel,
                                              const int* __restrict__ warp_tab,
                                              const unsigned short* __restrict__ col,
                                              const W* __restrict__ w,
                                              const float* __restrict__ x, int n_pre,
                                              int panel_width, float* __restrict__ sum, int* err,
                                              Wait&& wait) {
  extern __shared__ __align__(16) unsigned char anb_pc_smem[];
  __shared__ __align__(8) unsigned long long anb_pc_mbar;
  float* xs = reinterpret_cast<float*>(anb_pc_smem);
  const int p = cta_panel[blockIdx.x];
  const int c0 = p * panel_width;
  const int cw = min(panel_width, n_pre - c0);
  const int cw4 = cw & ~3;
  const int lane = threadIdx.x & 31;
  const int* wt = warp_tab + 3 * (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5));
  const int sb = wt[0], se = wt[1], hd = wt[2];
  const unsigned short* __restrict__ cp = col + 32ll * sb + lane;
  const W* __restrict__ wp = w + 32ll * sb + lane;
  unsigned short ca[U], cb[U];
  float wa[U], wb[U];
  // the U steps from step j: all of them (full) or those before se; a step
  // past the range reads as a padding header (no row), which ends the lane's
  // current row there; the range test is warp-uniform
  auto load = [&](unsigned short (&c)[U], float (&wv)[U], const int j) {
    const unsigned short* cq = cp + 32 * (j - sb);
    const W* wq = wp + 32 * (j - sb);
    if (j + U <= se) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        c[u] = __ldcs(cq + 32 * u);
        wv[u] = anb_pc_w(wq + 32 * u);
      }
    } else {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const bool in = j + u < se;
        c[u] = in ? __ldcs(cq + 32 * u) : (unsigned short)0xf000u;
        wv[u] = in ? anb_pc_w(wq + 32 * u) : 0.f;
      }
    }
  };
  float acc = 0.f;
  int cur = -1;                                      // sum index of the lane's current row
  auto consume = [&](const unsigned short (&c)[U], const float (&wv)[U]) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (c[u] >= 0xf000u) {                         // header: the previous slice ends
        if (cur >= 0) atomicAdd(&sum[cur], acc);
        acc = 0.f;
        cur = anb_pc_row(c[u], wv[u], w);
      } else {
        acc = fmaf(xs[c[u]], wv[u], acc);
      }
    }
  };
  if (sb < se) {                                     // in flight during the panel copy
    load(ca, wa, sb);
    if (hd < sb) cur = anb_pc_row(anb_ls_h(col + 32ll * hd + lane), anb_w1(w + 32ll * hd + lane), w);
  }
  wait();
  if (threadIdx.x == 0 && cw4 > 0) anb_bulk_issue(xs, x + c0, 4u * (unsigned)cw4, &anb_pc_mbar);
  for (int q = cw4 + threadIdx.x; q < cw; q += blockDim.x) xs[q] = x[c0 + q];
  __syncthreads();                                   // mbarrier and tail rates published
  if (cw4 > 0) anb_bulk_wait(&anb_pc_mbar, err);
  for (int j = sb; j < se; j += 2 * U) {
    load(cb, wb, j + U);
    consume(ca, wa);
    load(ca, wa, j + 2 * U);
    consume(cb, wb);
  }
  if (cur >= 0) atomicAdd(&sum[cur], acc);
}

// ---- event-driven transmission -----------------------------------------------------

// Exact gather: thread per post row; g[post] += w[j] for every synapse whose
// pre neuron spiked, in row (ascending pre) order.
template <typename R, typename W>
__device__ __forceinline__ void anb_spike_gather(int n_rows, const int* __restrict__ row_ptr,
                                                 const int* __restrict__ col,
                                                 const W* __restrict__ w,
                                                 const anb_u32* __restrict__ spk,
                                                 const int* __restrict__ post_rank,
                                                 R* __restrict__ g) {
  for (int row = blockIdx.x * blockDim.x + threadIdx.x; row < n_rows;
       row += gridDim.x * blockDim.x) {
    const int beg = row_ptr[row], end = row_ptr[row + 1];
    const int post = post_rank ? post_rank[row] : row;
    R acc = g[post];
    bool any = false;
    for (int j = beg; j < end; ++j) {
      if (anb_bit(spk, col[j])) {
        acc += (R)w[j];
        any = true;
      }
    }
    if (any) g[post] = acc;
  }
}

// Exact gather, warp per post row: lanes test 32 synapses at a time; the
// spiking ones are added in ascending pre rank (set bits of the ballot in
// order), which is the reference's per-post order.
template <typename R, typename W>
__device__ __forceinline__ void anb_spike_gather_warp(int n_rows, const int* __restrict__ row_ptr,
                                                      const int* __restrict__ col,
                                                      const W* __restrict__ w,
                                                      const anb_u32* __restrict__ spk,
                                                      const int* __restrict__ post_rank,
                                                      R* __restrict__ g) {
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int row = warp; row < n_rows; row += nwarps) {
    const int beg = row_ptr[row], end = row_ptr[row + 1];
    const int post = post_rank ? post_rank[row] : row;
    R acc = g[post];
    bool any = false;
    for (int base = beg; base < end; base += 32) {
      const int j = base + lane;
      const bool sp = j < end && anb_bit(spk, col[j]);
      anb_u32 m = __ballot_sync(0xffffffffu, sp);
      any |= m != 0u;
      const R wj = sp ? (R)w[j] : R(0);
      while (m) {
        const int b = __ffs(m) - 1;
        m &= m - 1;
        acc += __shfl_sync(0xffffffffu, wj, b);
      }
    }
    if (any && lane == 0) g[post] = acc;
  }
}

// Spike transmission with one delay per synapse (steps, 1..dmax): warp per
// post row; a spike emitted at step s reaches the synapses of delay t - s at
// step t. `ring` holds one spike bitmap of `words` words per step, `slots`
// steps. ORDERED adds the contributions one at a time in the reference's
// order: emission step ascending, then pre rank ascending (the push order of
// its ring of delayed spikes, ANNarchy/generator/Projection/SingleThread/
// LIL.py:915-969): a first pass over the row collects the delays that
// deliver a spike this step (a bit mask), then one pass per such delay, the
// largest first. Without ORDERED one pass adds them in pre-rank order.
template <typename R, typename W, bool ORDERED>
__device__ __forceinline__ void anb_spike_gather_delayed(int n_rows, const int* __restrict__ row_ptr,
                                                         const int* __restrict__ col,
                                                         const W* __restrict__ w,
                                                         const int* __restrict__ dly,
                                                         const anb_u32* __restrict__ ring, int words,
                                                         int slots, long long t,
                                                         const int* __restrict__ post_rank,
                                                         R* __restrict__ g) {
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int row = warp; row < n_rows; row += nwarps) {
    const int beg = row_ptr[row], end = row_ptr[row + 1];
    const int post = post_rank ? post_rank[row] : row;
    // delays (bit d) that deliver a spike to this row at step t
    unsigned long long dmask = 0ull;
    R acc = g[post];
    for (int base = beg; base < end; base += 32) {
      const int j = base + lane;
      bool sp = false;
      int d = 0;
      if (j < end) {
        d = dly[j];
        sp = anb_bit(ring + (size_t)anb_ring_slot(t - d, slots) * words, col[j]);
      }
      if (ORDERED) {
        unsigned long long m = sp ? (1ull << d) : 0ull;
        for (int o = 16; o > 0; o >>= 1) m |= __shfl_xor_sync(0xffffffffu, m, o);
        dmask |= m;
      } else {
        anb_u32 m = __ballot_sync(0xffffffffu, sp);
        dmask |= m;
        const R wj = sp ? (R)w[j] : R(0);
        while (m) {
          const int b = __ffs(m) - 1;
          m &= m - 1;
          acc += __shfl_sync(0xffffffffu, wj, b);
        }
      }
    }
    if (ORDERED) {
      for (unsigned long long rest = dmask; rest; ) {
        const int d = 63 - __clzll(rest);              // largest delay first: oldest spikes
        rest &= ~(1ull << d);
        const anb_u32* spk = ring + (size_t)anb_ring_slot(t - d, slots) * words;
        for (int base = beg; base < end; base += 32) {
          const int j = base + lane;
          const bool sp = j < end && dly[j] == d && anb_bit(spk, col[j]);
          anb_u32 m = __ballot_sync(0xffffffffu, sp);
          const R wj = sp ? (R)w[j] : R(0);
          while (m) {
            const int b = __ffs(m) - 1;
            m &= m - 1;
            acc += __shfl_sync(0xffffffffu, wj, b);
          }
        }
      }
    }
    if (dmask != 0ull && lane == 0) g[post] = acc;
  }
}

// ---- event-driven transmission in the reference's order (double precision) --------------
// A post neuron's conductance receives the step's increments one by one in
// ascending pre rank, but most post neurons receive none or one: instead of
// walking every row (anb_spike_gather_warp: 12 bytes per synapse and step),
// a deliver kernel walks the fan-out of the neurons that spiked and appends
// the position of each synapse reached to its post neuron's inbox (a counter
// and ANB_INBOX entries), and the update kernel sorts the few entries it
// finds and adds their weights in ascending order. A neuron with more
// entries than that walks its row as before. What bounds a step is then the
// latency of bitmap word -> column pointers -> synapse indices -> inbox
// atomics. Measured per step against the row-walking kernels: 100,000 neurons
// with 500 synapses each 139 -> 15.5 us, 10,000 neurons with 0.8M plastic
// synapses 22.8 -> 11.8 us, 3000 neurons with a delay per synapse 10.2 -> 8.3
// us (the last two are the launches and the chains of dependent loads). With
// what no kernel writes loaded before the wait for the previous kernel, and the
// bounds of a word's columns by a thread per neuron, the first two 13.8 and 9.6
// us; with the entries of all inboxes of a thread fetched at once, 11.4 and 9.6;
// with a plastic synapse's place in the inbox asked for before its statements,
// 8.4 for the plastic one. Steps with many spikes overfill the inboxes; then all
// rows are walked (the update kernels count spikes for this decision, which costs
// 0.1 to 0.5 us per step).
#define ANB_INBOX 8          // entries per post neuron: one 32-byte sector of 32-bit keys
#define ANB_DELIVER_WORDS 32 // bitmap words per CTA of a deliver kernel, at most
#define ANB_DELIVER_LIST (32 * ANB_DELIVER_WORDS)

// Lists the neurons whose bit is set in words [first, first + nw) of `bits`,
// whose word 0 is that of neuron 32 * w0 (nw <= ANB_DELIVER_WORDS), with the
// bounds ptr[row], ptr[row + 1] of their synapses (row = row_of[neuron], or
// the neuron itself without row_of; a negative row has none); returns their
// number. With slots > 0 `bits` is a ring of spike bitmaps (`stride` words per
// step) and the range repeats for the delays 1..slots: word i of it is word
// i % words of step t - d, d = i / words + 1, and the neuron's tag is d.
// list: 4 * ANB_DELIVER_LIST + 1 ints of shared memory (neurons, tags, begins,
// ends). Not inlined: modules call it once per projection, and its code is
// most of a deliver kernel's compile time.
__device__ __noinline__ int anb_list_spikes(int* list, const anb_u32* bits, int stride, int w0,
                                            int words, int slots, long long t, int first, int nw,
                                            const int* __restrict__ ptr,
                                            const int* __restrict__ row_of) {
  int* id = list;
  int* tag = list + ANB_DELIVER_LIST;
  int* beg = list + 2 * ANB_DELIVER_LIST;
  int* end = list + 3 * ANB_DELIVER_LIST;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < 32) {
    anb_u32 m = 0u;
    int base = 0, d = 0;
    if (lane < nw) {
      const int i = first + lane;
      d = slots > 0 ? i / words + 1 : 0;
      const int w = slots > 0 ? i % words : i;
      base = (w0 + w) << 5;
      m = slots > 0 ? bits[(size_t)anb_ring_slot(t - d, slots) * stride + w] : bits[w];
    }
    const int c = __popc(m);
    int incl = c;
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) list[4 * ANB_DELIVER_LIST] = incl;
    int k = incl - c;
    while (m) {
      id[k] = base + __ffs(m) - 1;
      tag[k++] = d;
      m &= m - 1;
    }
  }
  __syncthreads();
  const int n = list[4 * ANB_DELIVER_LIST];
  for (int e = threadIdx.x; e < n; e += blockDim.x) {
    const int r = row_of ? row_of[id[e]] : id[e];
    beg[e] = r < 0 ? 0 : ptr[r];
    end[e] = r < 0 ? 0 : ptr[r + 1];
  }
  __syncthreads();
  return n;
}

// The same from bounds that each thread has loaded beforehand (thread i: neuron
// i of the CTA's words; lane q holds word q, zero beyond): no load between the
// spikes and their synapses. Every warp counts for itself.
__device__ __forceinline__ int anb_list_ranges(int* list, anb_u32 words, int neuron, int beg, int end) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = __popc(words);
  const int n = __reduce_add_sync(0xffffffffu, c);
  const int before = __reduce_add_sync(0xffffffffu, lane < warp ? c : 0);
  const anb_u32 own = __shfl_sync(0xffffffffu, words, warp);
  if ((own >> lane) & 1u) {
    const int k = before + __popc(own & ((1u << lane) - 1u));
    list[k] = neuron;
    list[ANB_DELIVER_LIST + k] = 0;
    list[2 * ANB_DELIVER_LIST + k] = beg;
    list[3 * ANB_DELIVER_LIST + k] = end;
  }
  __syncthreads();
  return n;
}

// Runs body(neuron, tag, q) for every synapse q of the n listed neurons. All
// warps of the CTA share the synapses of a single spike, n of nwarps or more
// get one warp each, so that few loads wait for one another.
template <typename Body>
__device__ __forceinline__ void anb_for_spikes(const int* list, int n, Body body) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  int per = nwarps;
  while (per > 1 && per * n > nwarps) per >>= 1;
  const int groups = nwarps / per, sub = (warp % per) * 32 + lane;
  for (int e = warp / per; e < n && warp / per < groups; e += groups) {
    const int last = list[3 * ANB_DELIVER_LIST + e];
    for (int q = list[2 * ANB_DELIVER_LIST + e] + sub; q < last; q += 32 * per)
      body(list[e], list[ANB_DELIVER_LIST + e], q);
  }
}

// Spikes counted in the steps before t whose slots the ring holds (every step
// but t itself; the calling warp).
__device__ __forceinline__ anb_u32 anb_activity(const anb_u32* ring, int slots, long long t) {
  const int now = anb_ring_slot(t, slots);
  anb_u32 n = 0u;
  for (int q = threadIdx.x & 31; q < slots; q += 32)
    if (q != now) n += ring[q];
  return __reduce_add_sync(0xffffffffu, n);
}

// Appends `key` to the inbox of neuron `post` (entries beyond ANB_INBOX are
// only counted: the neuron then walks its row).
template <typename K>
__device__ __forceinline__ void anb_inbox_put(anb_u32* __restrict__ count, K* __restrict__ entry,
                                              int post, K key) {
  const anb_u32 slot = atomicAdd(&count[post], 1u);
  if (slot < ANB_INBOX) entry[(size_t)post * ANB_INBOX + slot] = key;
}

// g plus the weights of the 2 <= c <= ANB_INBOX synapses in the inbox of
// neuron i, in ascending key order (not inlined: rare, and long to compile).
template <typename R, typename K>
__device__ __noinline__ R anb_inbox_sorted(R g, anb_u32 c, const K* __restrict__ e,
                                           const R* __restrict__ w) {
  K k[ANB_INBOX];
#pragma unroll
  for (int a = 0; a < ANB_INBOX; ++a) k[a] = a < (int)c ? e[a] : ~K(0);
#pragma unroll 1
  for (int round = 0; round < ANB_INBOX / 2; ++round) {   // odd-even transposition sort
#pragma unroll
    for (int half = 0; half < 2; ++half)
#pragma unroll
      for (int a = half; a + 1 < ANB_INBOX; a += 2) {
        const K lo = k[a] < k[a + 1] ? k[a] : k[a + 1], hi = k[a] < k[a + 1] ? k[a + 1] : k[a];
        k[a] = lo;
        k[a + 1] = hi;
      }
  }
  R v[ANB_INBOX];
#pragma unroll
  for (int a = 0; a < ANB_INBOX; ++a) v[a] = a < (int)c ? w[(anb_u32)k[a]] : R(0);
#pragma unroll
  for (int a = 0; a < ANB_INBOX; ++a)
    if (a < (int)c) g += v[a];
  return g;
}

// The same for 0 <= c <= ANB_INBOX; the low 32 bits of a key are the
// synapse's position in w (with delays the high bits order the emission
// steps, oldest first).
template <typename R, typename K>
__device__ __forceinline__ R anb_inbox_add(R g, anb_u32 c, const K* __restrict__ entry, int i,
                                           const R* __restrict__ w) {
  const K* __restrict__ e = entry + (size_t)i * ANB_INBOX;
  if (c == 1u) return g + w[(anb_u32)e[0]];
  return c ? anb_inbox_sorted<R, K>(g, c, e, w) : g;
}

// The first two entries of neuron i's inbox.
__device__ __forceinline__ void anb_inbox_first(const anb_u32* __restrict__ entry, int i, anb_u32& a, anb_u32& b) {
  const uint2 e = *reinterpret_cast<const uint2*>(entry + (size_t)i * ANB_INBOX);
  a = e.x;
  b = e.y;
}
__device__ __forceinline__ void anb_inbox_first(const unsigned long long* __restrict__ entry, int i,
                                                unsigned long long& a, unsigned long long& b) {
  const ulonglong2 e = *reinterpret_cast<const ulonglong2*>(entry + (size_t)i * ANB_INBOX);
  a = e.x;
  b = e.y;
}

// Rows walked in the reference's order: the conductance g plus the weights w[j] of
// the row's synapses whose pre neuron's bit is set, in ascending pre rank. Loads of
// U steps are issued together, so that a long row is not a chain of trips to L2.
// (All rows walked, 1000 neurons with 1000 synapses each, 5 % spiking: U = 4, 2, 1
// 11.2, 13.1, 18.7 us per step; a kernel of its own without U 18.5. The update
// kernels, where few neurons' inboxes run over, take U = 1: with more in flight
// their other code slowed down, 11.9 instead of 11.6 us per step of 100,000 neurons
// with 500 synapses each.) Whole warp, one row. Not inlined: half the compile time.
template <typename R, int U>
__device__ __noinline__ R anb_row_gather(R g, int beg, int end, const int* __restrict__ col,
                                         const R* __restrict__ w, const anb_u32* bits) {
  const int lane = threadIdx.x & 31;
  for (int base = beg; base < end; base += 32 * U) {
    int c[U];
    bool sp[U];
    R v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) c[u] = base + 32 * u + lane < end ? col[base + 32 * u + lane] : -1;
#pragma unroll
    for (int u = 0; u < U; ++u) sp[u] = c[u] >= 0 && anb_bit(bits, c[u]);
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = sp[u] ? w[base + 32 * u + lane] : R(0);
#pragma unroll
    for (int u = 0; u < U; ++u)
      for (anb_u32 m = __ballot_sync(0xffffffffu, sp[u]); m; m &= m - 1)
        g += __shfl_sync(0xffffffffu, v[u], __ffs(m) - 1);
  }
  return g;
}

// One row per lane (lanes on their own): four and more overflowing neurons of a
// warp. (32 rows of 1000 synapses one after another took 207 us, this way 104.)
template <typename R>
__device__ __noinline__ R anb_lane_gather(R g, int beg, int end, const int* __restrict__ col,
                                          const R* __restrict__ w, const anb_u32* bits) {
  constexpr int U = 4;
  for (int base = beg; base < end; base += U) {
    int c[U];
    bool sp[U];
    R v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) c[u] = base + u < end ? col[base + u] : -1;
#pragma unroll
    for (int u = 0; u < U; ++u) sp[u] = c[u] >= 0 && anb_bit(bits, c[u]);
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = sp[u] ? w[base + u] : R(0);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (sp[u]) g += v[u];
  }
  return g;
}

// The same with one delay per synapse: emission steps t - slots .. t - 1 in
// order, ascending pre rank within each: one pass over the row for the delays
// that deliver a spike in step t, then one for each of them. The ring slot of the
// oldest step is read from `oldest` (the update kernels of step t write that
// slot: they keep a copy).
struct anb_delay_ring {
  const anb_u32 *ring, *oldest;
  int words, slots, now;                               // now: the slot of step t
  __device__ __forceinline__ const anb_u32* at(int d) const {
    return d == slots ? oldest : ring + (size_t)(now - d < 0 ? now - d + slots : now - d) * words;
  }
};

template <typename R, int U>
__device__ __noinline__ R anb_row_gather_delayed(R g, int beg, int end, const int* __restrict__ col,
                                                 const R* __restrict__ w,
                                                 const int* __restrict__ dly, const anb_delay_ring q) {
  const int lane = threadIdx.x & 31;
  anb_u32 lo = 0u, hi = 0u;                            // the delays that deliver
  for (int base = beg; base < end; base += 32 * U) {
    int c[U], d[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int j = base + 32 * u + lane;
      c[u] = j < end ? col[j] : -1;
      d[u] = j < end ? dly[j] : 0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (c[u] >= 0 && anb_bit(q.at(d[u]), c[u])) {
        if (d[u] < 32) lo |= 1u << d[u];
        else hi |= 1u << (d[u] - 32);
      }
  }
  lo = __reduce_or_sync(0xffffffffu, lo);
  hi = __reduce_or_sync(0xffffffffu, hi);
  for (unsigned long long rest = (unsigned long long)hi << 32 | lo; rest;) {
    const int at = 63 - __clzll(rest);
    rest &= ~(1ull << at);
    const anb_u32* bits = q.at(at);
    for (int base = beg; base < end; base += 32 * U) {
      int c[U];
      bool sp[U];
      R v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int j = base + 32 * u + lane;
        c[u] = j < end && dly[j] == at ? col[j] : -1;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) sp[u] = c[u] >= 0 && anb_bit(bits, c[u]);
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = sp[u] ? w[base + 32 * u + lane] : R(0);
#pragma unroll
      for (int u = 0; u < U; ++u)
        for (anb_u32 m = __ballot_sync(0xffffffffu, sp[u]); m; m &= m - 1)
          g += __shfl_sync(0xffffffffu, v[u], __ffs(m) - 1);
    }
  }
  return g;
}

template <typename R>
__device__ __noinline__ R anb_lane_gather_delayed(R g, int beg, int end, const int* __restrict__ col,
                                                  const R* __restrict__ w,
                                                  const int* __restrict__ dly, anb_delay_ring q) {
  unsigned long long rest = 0ull;
#pragma unroll 4
  for (int j = beg; j < end; ++j) {
    const int d = dly[j];
    if (anb_bit(q.at(d), col[j])) rest |= 1ull << d;
  }
  while (rest) {
    const int at = 63 - __clzll(rest);
    rest &= ~(1ull << at);
    const anb_u32* bits = q.at(at);
#pragma unroll 4
    for (int j = beg; j < end; ++j)
      if (dly[j] == at && anb_bit(bits, col[j])) g += w[j];
  }
  return g;
}

// Fast scatter: a warp per 32-neuron bitmap word of the pre population
// (words [w0, w1)); for every set bit the warp walks that neuron's outgoing
// synapses (pre-major: col_ptr / post_idx / w_pre) and adds w to g[post]
// with atomics. Warp-uniform control flow; lanes stride the fan-out. This CTA
// is number blk of the nblk that share the words.
template <typename R, typename W>
__device__ __forceinline__ void anb_spike_scatter(int w0, int w1, const anb_u32* __restrict__ spk,
                                                  const int* __restrict__ col_ptr,
                                                  const int* __restrict__ post_idx,
                                                  const W* __restrict__ w_pre,
                                                  R* __restrict__ g, int blk, int nblk) {
  const int lane = threadIdx.x & 31;
  const int warp = (int)(blk * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (int)(nblk * blockDim.x) >> 5;
  for (int word = w0 + warp; word < w1; word += nwarps) {
    anb_u32 m = spk[word];
    while (m) {
      const int b = __ffs(m) - 1;
      m &= m - 1;
      const int pre = (word << 5) + b;
      const int beg = col_ptr[pre], end = col_ptr[pre + 1];
      for (int k = beg + lane; k < end; k += 32) atomicAdd(&g[post_idx[k]], (R)anb_wf(w_pre[k]));
    }
  }
}

// ---- thread-block clusters (distributed shared memory) ----------------------------------
// The cluster engine splits a network's neurons over the CTAs of one
// cluster; spikes are delivered into the owning CTA's shared memory with
// DSMEM reductions and the CTAs meet at one hardware cluster barrier per
// step (no spin loop).

__device__ __forceinline__ unsigned anb_cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

__device__ __forceinline__ unsigned anb_smem_addr(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}

// Address of the same shared-memory offset in CTA `rank` of the cluster.
__device__ __forceinline__ unsigned anb_cluster_map(unsigned addr, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

__device__ __forceinline__ void anb_cluster_red_add(unsigned addr, float v) {
  asm volatile("red.relaxed.cluster.shared::cluster.add.f32 [%0], %1;" ::"r"(addr), "f"(v)
               : "memory");
}

__device__ __forceinline__ void anb_cluster_st_u32(unsigned addr, anb_u32 v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

__device__ __forceinline__ void anb_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::
                   : "memory");
}

// mbarriers of this CTA (shared-memory addresses): `count` arrivals per phase,
// one of them with the bytes to expect from the cluster's other CTAs.
__device__ __forceinline__ void anb_mbar_init(unsigned bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void anb_mbar_expect(unsigned bar, unsigned bytes) {
  asm volatile("{ .reg .b64 st; mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1; }"
               ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void anb_mbar_arrive(unsigned bar) {
  asm volatile("{ .reg .b64 st; mbarrier.arrive.shared::cta.b64 st, [%0]; }" ::"r"(bar) : "memory");
}
// Bounded wait (about a second) for the phase of the given parity; false and
// an error code when it ran out. Polls without suspending: the phases are a
// few hundred cycles apart.
__device__ __forceinline__ bool anb_mbar_wait(unsigned bar, unsigned parity, int* err) {
  unsigned done = 0;
  long long c0 = 0;
  for (int it = 1;; ++it) {
    asm volatile(
        "{ .reg .pred p; mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
        : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    if (done) return true;
    if ((it & 1023) == 0) {
      const long long c = clock64();
      if (c0 == 0) c0 = c;
      if (c - c0 > 2000000000ll) {
        anb_report(err, ANB_DEVERR_BARRIER_TIMEOUT);
        return false;
      }
    }
  }
}

// Appends the values v of the lanes with `in` to a list of *n entries.
__device__ __forceinline__ void anb_pack(anb_u32 v, bool in, anb_u32* list, int* n) {
  const unsigned z = __ballot_sync(0xffffffffu, in);
  if (in) list[*n + __popc(z & ((1u << (threadIdx.x & 31)) - 1u))] = v;
  *n += __popc(z);
}
// g plus w once for every one of the n listed masks with this lane's bit (the
// list is 16-byte aligned and padded to a multiple of 4 with zeros).
template <typename R>
__device__ __forceinline__ R anb_mask_add(R g, R w, const anb_u32* list, int n) {
  const anb_u32 bit = 1u << (threadIdx.x & 31);
#pragma unroll 1
  for (int k = 0; k < n; k += 4) {
    const uint4 v = *reinterpret_cast<const uint4*>(list + k);
    if (v.x & bit) g += w;
    if (v.y & bit) g += w;
    if (v.z & bit) g += w;
    if (v.w & bit) g += w;
  }
  return g;
}
// The same with one delay per synapse: for every listed mask with this lane's
// bit, one event more for the step its delay names. at[k]: the projection << 24
// plus the position of the delays: of the first of the mask's synapses (PACKED),
// or the row of a matrix whose column of this lane `delays` is (`stride` bytes
// per row). cnt: 16-bit counters, `chunk` per step in a ring of `slots`,
// `proj_size` per projection; `from`: the slot of the emission step. A delay
// below `least` has arrived before the run began. The counters take an atomic
// without a result: nothing waits for it (load, add and store one after another
// were 35 cycles per mask).
template <bool PACKED>
__device__ __forceinline__ void anb_mask_delays(const anb_u32* list, const anb_u32* at, int n,
                                                const unsigned char* delays, int stride, anb_u32* cnt,
                                                int proj_size, int chunk, int from, int slots, int least) {
  constexpr int U = PACKED ? 4 : 8;         // (a matrix in global memory: more loads under way)
  const int lane = threadIdx.x & 31;
  const anb_u32 bit = 1u << lane, below = bit - 1u, one = (lane & 1) ? 0x10000u : 1u;
#pragma unroll 1
  for (int k = 0; k < n; k += U) {
    anb_u32 m[U], q[U];
    int d[U];
#pragma unroll
    for (int u = 0; u < U; u += 4) {
      const uint4 v = *reinterpret_cast<const uint4*>(list + k + u);
      const uint4 r = *reinterpret_cast<const uint4*>(at + k + u);
      m[u] = v.x; m[u + 1] = v.y; m[u + 2] = v.z; m[u + 3] = v.w;
      q[u] = r.x; q[u + 1] = r.y; q[u + 2] = r.z; q[u + 3] = r.w;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const anb_u32 p = q[u] & 0xffffffu;
      d[u] = !(m[u] & bit) ? 0 : PACKED ? (int)delays[p + __popc(m[u] & below)] : (int)delays[(size_t)p * stride];
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (d[u] > 0 && d[u] >= least) {
        const int s = from + d[u] >= slots ? from + d[u] - slots : from + d[u];
        atomicAdd(cnt + ((int)(q[u] >> 24) * proj_size + s * chunk + (int)threadIdx.x) / 2, one);
      }
  }
}
// g plus w as often as counted; the counter starts again.
template <typename R>
__device__ __forceinline__ R anb_mask_drain(R g, R w, unsigned short* cnt) {
  int c = *cnt;
  if (c) *cnt = 0;
  if (c > 0) g += w;                        // (mostly none or one: no vote to wait for)
  if (c > 1) g += w;
  for (c -= 2; __any_sync(0xffffffffu, c > 0); --c)
    if (c > 0) g += w;
  return g;
}
// The same without votes (lanes on their own).
template <typename R>
__device__ __forceinline__ R anb_count_add(R g, R w, unsigned short* cnt) {
  int c = *cnt;
  if (c) {
    *cnt = 0;
    do g += w;
    while (--c);
  }
  return g;
}
// Store of one word into another CTA of the cluster, counted on that CTA's
// mbarrier (launches with a cluster only; the own CTA's word is an ordinary
// store).
__device__ __forceinline__ void anb_st_async(unsigned addr, anb_u32 v, unsigned bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.u32 [%0], %1, [%2];"
               ::"r"(addr), "r"(v), "r"(bar) : "memory");
}

// Fast scatter from a spike list: work item = (spike, 32-synapse chunk of its
// fan-out), so a warp does one pass per item whatever the fan-out; spikes
// outside [lo, hi) (not pre neurons of this projection) are skipped.
template <typename R, typename W>
__device__ __forceinline__ void anb_spike_scatter_list(int lo, int hi, const int* __restrict__ list,
                                                       int count, int chunks,
                                                       const int* __restrict__ col_ptr,
                                                       const int* __restrict__ post_idx,
                                                       const W* __restrict__ w_pre,
                                                       R* __restrict__ g, int blk, int nblk) {
  const int lane = threadIdx.x & 31;
  const long long items = (long long)count * chunks;
  for (long long it = (blk * blockDim.x + threadIdx.x) >> 5; it < items;
       it += (nblk * blockDim.x) >> 5) {
    const int pre = list[it / chunks];
    if (pre < lo || pre >= hi) continue;
    const int c = (int)(it % chunks);
    const int end = col_ptr[pre + 1];
    for (int q = col_ptr[pre] + c * 32 + lane; q < end; q += 32 * chunks)
      atomicAdd(&g[post_idx[q]], (R)anb_wf(w_pre[q]));
  }
}

// ---- grid-wide barrier of a cooperative persistent launch ----------------------------
// bar[0] counts the CTAs that arrived, bar[1] is the generation. Every CTA
// reads the generation before arriving; the last to arrive resets the count
// and advances the generation, the others wait (bounded by a cycle budget of
// about one second) until it changes. Returns false when this or any other
// CTA gave up (err[0] holds ANB_DEVERR_BARRIER_TIMEOUT): the caller leaves its
// loop. Other device errors (a full monitor ring) do not stop the run.
#define ANB_GRID_WAIT_CYCLES (2000000000ll)
__device__ __forceinline__ bool anb_grid_sync(unsigned* bar, int* err) {
  __shared__ int anb_gs_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile unsigned* gen = bar + 1;
    const unsigned g = *gen;
    __threadfence();
    const unsigned arrived = atomicAdd(bar, 1u);
    int ok = 1;
    if (arrived == gridDim.x - 1) {
      atomicExch(bar, 0u);
      __threadfence();
      atomicAdd(bar + 1, 1u);
    } else {
      const long long c0 = clock64();
      while (*gen == g) {
        if (clock64() - c0 > ANB_GRID_WAIT_CYCLES ||
            *(volatile int*)err == ANB_DEVERR_BARRIER_TIMEOUT) {
          ok = 0;
          break;
        }
        __nanosleep(64);
      }
      if (!ok) atomicExch(err, ANB_DEVERR_BARRIER_TIMEOUT);
    }
    __threadfence();
    anb_gs_ok = ok && *(volatile int*)err != ANB_DEVERR_BARRIER_TIMEOUT;
  }
  __syncthreads();
  return anb_gs_ok != 0;
}

// ---- rate-coded networks that stay on chip -------------------------------------------------
// A CTA keeps the incoming synapses of its neurons in shared memory, as items
// of ROWS rows (one warp at a time) with LANES lanes per row: step m of an
// item holds element m * LANES + g of row q at position q * LANES + g, so a
// warp's loads of weights and columns are conflict-free; the rates are
// gathered from the CTA's copy. What bounds a step: in double precision the
// chain of ordered additions of a row (the loads of UNROLL steps are issued
// ahead of it), the exchange of the rates and the barrier.

// Fills a projection's part of the CTA's pool: rb = (first element of the part
// in ri, its elements, its place in the pool), ri = each element's place in
// the CSR arrays; -1 (past a row's end) gets weight 0 and column `pad`, where
// the CTA's copy of the rates holds a zero.
template <typename W>
__device__ __noinline__ void anb_rate_fill(const int* __restrict__ rb, const int* __restrict__ ri,
                                              const int* __restrict__ col, const W* __restrict__ w,
                                              int pad, W* pool_w, unsigned short* pool_c) {
  const int* __restrict__ src = ri + rb[0];
  const int n = rb[1], at = rb[2];
#pragma unroll 2
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    const int j = src[k];
    pool_w[at + k] = j >= 0 ? w[j] : W(0);
    pool_c[at + k] = (unsigned short)(j >= 0 ? col[j] : pad);
  }
}

// Loads from shared-memory addresses (volatile: not moved across barriers).
__device__ __forceinline__ void anb_lds(unsigned a, float* v) {
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(*v) : "r"(a));
}
__device__ __forceinline__ void anb_lds(unsigned a, double* v) {
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(*v) : "r"(a));
}
__device__ __forceinline__ void anb_lds(unsigned a, unsigned short* v) {
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(*v) : "r"(a));
}

// Weighted sum of the calling lane's row of one item (all lanes of the row
// get it; whole warp): blocks of U steps, the columns loaded two blocks and
// the rates and weights one block ahead of the additions. Double precision:
// one lane, stored order, bound by the chain of additions (9 cycles each); a
// padding element adds +0, which changes no sum. The columns' loads may run
// two blocks past the item (inside the CTA's pool, which is that much longer).
// Pool and rates as shared-memory addresses; not inlined (a network calls it
// once per projection, and its code is most of the module's compile time).
template <typename R, typename W, int LANES, int ROWS>
__device__ __noinline__ R anb_rate_row(int first, int steps, unsigned pool_w, unsigned pool_c, unsigned x) {
  constexpr int U = LANES == 1 ? 8 : 4, L = ROWS * LANES;
  const int lane = threadIdx.x & 31;
  const int at = first + (lane < L ? lane : 0);
  unsigned w = pool_w + (unsigned)(at * sizeof(W)), c = pool_c + 2u * at;
  // single precision: fused products in two sums (a product rounded by itself and
  // one sum were 1.1 to 1.3 times as far from 64 bits; the launch plan fuses too)
  constexpr bool F = sizeof(R) == 4;
  R s = R(0), s1 = R(0), p[U], q[U];
  auto keep = [&](const R (&x)[U], const W (&v)[U]) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      q[u] = (R)anb_wf(v[u]);
      p[u] = F ? x[u] : x[u] * q[u];
    }
  };
  auto add = [&]() {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (!F) s += p[u];
      else if (u < U / 2) s = fma(p[u], q[u], s);
      else s1 = fma(p[u], q[u], s1);
    }
  };
  if (steps > 0) {
    unsigned short cn[U];
    R xn[U];
    W wn[U];
#pragma unroll
    for (int u = 0; u < U; ++u) anb_lds(c + 2u * u * L, &cn[u]);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      anb_lds(x + (unsigned)sizeof(R) * cn[u], &xn[u]);
      anb_lds(w + (unsigned)sizeof(W) * u * L, &wn[u]);
      anb_lds(c + 2u * (U + u) * L, &cn[u]);
    }
    keep(xn, wn);
#pragma unroll 1
    for (int m = U; m < steps; m += U) {
      w += (unsigned)sizeof(W) * U * L;
      c += 2u * U * L;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        anb_lds(x + (unsigned)sizeof(R) * cn[u], &xn[u]);
        anb_lds(w + (unsigned)sizeof(W) * u * L, &wn[u]);
        anb_lds(c + 2u * (U + u) * L, &cn[u]);
      }
      add();
      keep(xn, wn);
    }
    add();
  }
  if (F) s += s1;
#pragma unroll
  for (int o = LANES / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

__device__ __forceinline__ void anb_cluster_st(unsigned addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void anb_cluster_st(unsigned addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}

// Grid-wide barrier on a counter that only grows (zero at the launch): the
// CTA's arrival, then a bounded wait until `target` arrivals. Returns false
// when this or another CTA gave up (see anb_grid_sync).
__device__ __forceinline__ bool anb_grid_meet(unsigned* bar, unsigned target, int* err) {
  __shared__ int anb_gm_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    // the release covers the CTA's writes: the CTA barrier orders them before it
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
    int ok = 1;
    unsigned v = 0;
    const long long c0 = clock64();
    for (int it = 0;; ++it) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
      if ((int)(v - target) >= 0) break;
      if ((it & 63) == 63 && (clock64() - c0 > ANB_GRID_WAIT_CYCLES ||
                              *(volatile int*)err == ANB_DEVERR_BARRIER_TIMEOUT)) {
        ok = 0;
        break;
      }
    }
    if (!ok) atomicExch(err, ANB_DEVERR_BARRIER_TIMEOUT);
    anb_gm_ok = ok;
  }
  __syncthreads();
  return anb_gm_ok != 0;
}

// ---- monitors ---------------------------------------------------------------------------

// Copy n values (converted to double) into slot `slot` of a ring of `cap` slots.
template <typename T>
__device__ __forceinline__ void anb_record(const T* __restrict__ src, const int* __restrict__ ranks,
                                           int n, double* __restrict__ buf, long long slot) {
  double* dst = buf + slot * (long long)n;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x)
    dst[k] = (double)src[ranks ? ranks[k] : k];
}


// Exclusive prefix sum of x over the CTA (blockDim.x a multiple of 32, at
// most 1024). `warp_sums` is 32 ints of shared memory; two CTA barriers.
__device__ __forceinline__ int anb_block_exclusive_scan(int x, int* warp_sums, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int incl = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int s = lane < nw ? warp_sums[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += v;
    }
    if (lane < nw) warp_sums[lane] = s;
  }
  __syncthreads();
  *total = warp_sums[nw - 1];
  return (warp ? warp_sums[warp - 1] : 0) + incl - x;
}
