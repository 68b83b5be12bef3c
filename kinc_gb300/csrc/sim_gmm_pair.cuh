/*
 * sim_gmm_pair.cuh -- GMM clustering with one warp per gene pair.
 *
 * GMM::fit (src/core/pairwise_gmm.cpp:367-445) sums every quantity of an EM
 * iteration in sample order, but what it sums -- log-densities, exponentials,
 * products -- is independent from sample to sample.  So the warp computes the
 * terms of 64 samples at a time (two per lane, in packed FP32), lays them out
 * in shared memory as one row per accumulator, and then every accumulator is
 * summed in sample order by a lane of its own: 3K + 1 rows after the E step
 * (responsibility sums, mean sums, log-likelihood) and 3K for the covariances.
 * Each value is formed by the operations of gmm_fit (sim_device.cuh) in their
 * order, so the results are the same bits.
 *
 * Against one pair per lane (k_similarity): a pair's working set (X, log p(x)
 * and the K x N responsibilities, 32 bytes per sample at K = 5) stays in
 * shared memory or L2 instead of streaming 21 MB per pair through HBM, about
 * 10 pairs fill an SM instead of 640, and a small block of pairs finishes in
 * the latency of one cooperative fit instead of one lane's.  GMM k <= 5 (BIC,
 * outliers, Spearman), tile kernel -> this one: 1,128 pairs of 96 samples
 * 71.8 -> 1.9 ms, 32,768 pairs of 1,000 samples (N = 810) 580 -> 173 ms,
 * 131,072 pairs 1,131 -> 682 ms, 196,608 pairs of 500 samples (ICL, both
 * correlations) 947 -> 561 ms.
 *
 * What bounds it: per 64 samples, component and iteration the fit needs 122
 * cycles of a scheduler's FP32 pipe (a packed FP32 instruction takes two; the
 * three exponentials are half of it) and the ordered sums 128 per fit; at K = 5
 * and N = 832 that is 192 cycles per SM and chunk of 64 samples, 59 % of the 323
 * measured with 11 pairs per SM.  (Over a whole block, with its other K, sorts and
 * waits, the counters show the FP32 pipe busy 43 % of the time.)  The shared-memory pipe carries 26 wavefronts per component
 * beside it.
 */
#pragma once

#include "sim_pair.cuh"

#include <type_traits>

namespace kinc {

constexpr int GP_WARPS = 16;                /* warps (pairs) per SM at most: 128 registers each */
constexpr int GP_WARPS_FEW = 12;            /* at most, where no more pairs fit an SM: 168 registers each */
/* fewer pairs than this an SM with vg in shared memory: it moves to global memory */
__host__ __device__ constexpr int gp_shared_pairs(int warps)
{
   return warps == GP_WARPS_FEW ? 9 : 13;
}
constexpr int GP_CHUNK = 64;                /* samples the warp computes in one packed operation, and lays out
                                               as term rows together */
constexpr int GP_ROW = GP_CHUNK + 4;        /* floats of a term row: rows start 4 banks apart, so the 16-byte
                                               reads of 8 lanes on 8 rows touch all 32 banks once */
constexpr int GP_KMAX = 5;                  /* largest component count compiled */
constexpr int GP_PAR = 16;                  /* floats of one component's published parameters: m0, m1, the inverse
                                               covariance's a, b, c, the normaliser, log(pi), the largest
                                               log(gamma/pi), each twice (both halves of a packed operand) */

/* floats of shared memory one pair needs: n usable samples at most, fits of up to max_k components (their
 * log(gamma/pi) in shared memory or, with `global`, not), sort_rows rows of next_pow2(n) floats for the
 * outlier (1) and Spearman (2) networks, which reuse the fit's arrays */
__host__ __device__ inline int gp_slot_floats(int n, int max_k, int sort_rows, bool global)
{
   const int n64 = (n + GP_CHUNK - 1) / GP_CHUNK * GP_CHUNK;
   int p2 = 2;
   while ( p2 < n ) p2 *= 2;
   const int fit = n64 + 32 + (global ? 0 : max_k * n64) + 2 * 3 * max_k * GP_ROW;
   const int sort = sort_rows * p2;
   return (2 * n64 + (fit > sort ? fit : sort) + GP_KMAX * GP_PAR + 31) & ~31;
}

/* floats of vg of one pair in global memory */
__host__ __device__ inline int gp_global_floats(int n, int max_k)
{
   return max_k * (((n > 0 ? n : 1) + GP_CHUNK - 1) / GP_CHUNK * GP_CHUNK);
}

/* one pair's arrays in shared memory */
struct GpView
{
   float* x;          /* sample pairs (2i, 2i+1) as { x0, x0', x1, x1' } */
   float* lpx;        /* log p(x), one per sample; starts on the bank its summing lane leaves free */
   float* vg;         /* [k][n64]: log-density, then log(gamma/pi) after E, gamma/pi after M1 */
   float* terms;      /* term rows of two chunks, 3K rows each */
   float* par;        /* [k][GP_PAR] */
   float* work;       /* lpx, vg and terms as one buffer (sorts, work labels) */
   float nz;          /* -0 */
   int n64, N, nch;   /* row length, usable samples, chunks in use */
};

/* the same as offsets (floats) into the CTA's shared memory, for calls that are not inlined: a pointer
 * argument would lose its address space */
struct GpLayout
{
   float* vg_global;  /* vg when it lies in global memory */
   int x, lpx, vg, terms, par;
   int n64, N, nch;
   float nz;
   __device__ __forceinline__ GpView view() const
   {
      extern __shared__ __align__(16) float gp_shared[];
      GpView s;
      s.x = gp_shared + x;
      s.lpx = gp_shared + lpx;
      s.vg = gp_shared + vg;
      s.terms = gp_shared + terms;
      s.par = gp_shared + par;
      s.work = s.terms;
      s.nz = nz;
      s.n64 = n64;
      s.N = N;
      s.nch = nch;
      return s;
   }
};

__device__ __forceinline__ float2 gp_x(const GpView& s, int i)
{
   const float* q = s.x + (i >> 1) * 4 + (i & 1);
   return make_float2(q[0], q[2]);
}

/* the samples as the outlier and correlation passes read them */
struct GpSamples
{
   GpView s;
   __device__ __forceinline__ float2 operator()(int i) const { return gp_x(s, i); }
};

__device__ __forceinline__ F2 gp_ld2(const float* p)
{
   F2 r;
   r.v = *reinterpret_cast<const unsigned long long*>(p);
   return r;
}

__device__ __forceinline__ void gp_st2(float* p, F2 v)
{
   *reinterpret_cast<unsigned long long*>(p) = v.v;
}

/* vg in shared memory, or (G) in global memory, past the first-level cache it would not fit */
template <bool G>
__device__ __forceinline__ F2 gp_ldv(const float* p)
{
   F2 r;
   if ( G )
      r.v = __ldcg(reinterpret_cast<const unsigned long long*>(p));
   else
      r.v = *reinterpret_cast<const unsigned long long*>(p);
   return r;
}

template <bool G>
__device__ __forceinline__ void gp_stv(float* p, F2 v)
{
   if ( G )
      __stcg(reinterpret_cast<unsigned long long*>(p), v.v);
   else
      *reinterpret_cast<unsigned long long*>(p) = v.v;
}

/* the largest of the lanes' values, none of them NaN: floats ordered as integers */
__device__ __forceinline__ float gp_warp_max(float v)
{
   const int b = __float_as_int(v);
   const int m = __reduce_max_sync(0xffffffffu, b ^ ((b >> 31) & 0x7fffffff));
   return __int_as_float(m ^ ((m >> 31) & 0x7fffffff));
}

/* the polynomial of kinc_expf on both halves (kinc_fmath.h) */
__device__ __forceinline__ F2 gp_exp_poly(F2 x, F2 n)
{
   F2 r = fma2(n, f2(-KINC_F_LN2_HI), x);
   r = fma2(n, f2(-KINC_F_LN2_LO), r);
   F2 p = f2(KINC_EXP_C6);
   p = fma2(p, r, f2(KINC_EXP_C5));
   p = fma2(p, r, f2(KINC_EXP_C4));
   p = fma2(p, r, f2(KINC_EXP_C3));
   p = fma2(p, r, f2(KINC_EXP_C2));
   p = fma2(p, r, f2(1.0f));
   return fma2(p, r, f2(1.0f));
}

/* p * 2^n by the exponent field, n in the low bits of the shifted sum */
__device__ __forceinline__ F2 gp_scale(F2 p, F2 shifted)
{
   float p0, p1, s0, s1;
   split(p, p0, p1);
   split(shifted, s0, s1);
   return f2(__uint_as_float(__float_as_uint(p0) + (__float_as_uint(s0) << 23)),
             __uint_as_float(__float_as_uint(p1) + (__float_as_uint(s1) << 23)));
}

__device__ __forceinline__ F2 gp_clamp(F2 x, float lo)
{
   float a, b;
   split(x, a, b);
   return f2(fmaxf(a, lo), fmaxf(b, lo));
}

/*
 * kinc_expf on both halves for finite x <= 70, without branches: the result is formed 2^26 too
 * large, where it is a normal float for every x >= -105, and scaled back with one rounding -- exact
 * for normal results, the single rounding of kinc_expf_tail for subnormal ones; below -105 the
 * result is zero either way.  (The shift of 26 rides in the rounding constant.)
 */
__device__ __forceinline__ F2 gp_exp(F2 x)
{
   x = gp_clamp(x, -105.0f);
   const F2 shifted = fma2(x, f2(KINC_F_LOG2E), f2(12582912.0f + 26.0f));
   const F2 n = shifted - f2(12582912.0f + 26.0f);
   return gp_scale(gp_exp_poly(x, n), shifted) * f2(1.4901161193847656e-08f);   /* 2^-26 */
}

/*
 * kinc_expf for finite x <= 0 whose results are summed with an exp(0) = 1 of at most four others:
 * anything below e^-86 leaves that sum as it is (a partial sum without the 1 either exceeds 2^-75 and
 * absorbs it, or is absorbed by the 1), so x is cut off there and every result is a normal float.
 */
__device__ __forceinline__ F2 gp_exp_beside_one(F2 x)
{
   x = gp_clamp(x, -86.0f);
   const F2 shifted = fma2(x, f2(KINC_F_LOG2E), f2(12582912.0f));
   const F2 n = shifted - f2(12582912.0f);
   return gp_scale(gp_exp_poly(x, n), shifted);
}

__device__ __forceinline__ F2 gp_exp_any(F2 x)
{
   float a, b;
   split(x, a, b);
   return f2(kinc_expf(a), kinc_expf(b));
}

/* kinc_logf's reduction table, one entry per lane */
struct GpLogTable
{
   float inv, hi, lo;
   __device__ __forceinline__ void load(int lane)
   {
      const kinc_log_entry t = kinc_log_table_d[lane];
      inv = t.inv;
      hi = t.hi;
      lo = t.lo;
   }
};

/* kinc_logf of a positive normal float; every lane of the warp calls it */
__device__ __forceinline__ float gp_log(float x, const GpLogTable& t)
{
   const uint32_t b = __float_as_uint(x);
   const uint32_t tmp = b - 0x3f340000u;
   const int e = (int)tmp >> 23;
   const int i = (int)(tmp >> 18);
   const float m = __uint_as_float(b - (tmp & 0xff800000u));
   const float inv = __shfl_sync(0xffffffffu, t.inv, i);
   const float thi = __shfl_sync(0xffffffffu, t.hi, i);
   const float tlo = __shfl_sync(0xffffffffu, t.lo, i);
   const float z = fmaf(m, inv, -1.0f);
   float q = 0.2f;
   q = fmaf(q, z, -0.25f);
   q = fmaf(q, z, 0.333333343267440796f);
   q = fmaf(q, z, -0.5f);
   const float z2 = z * z;
   const float ef = (float)e;
   const float hi = fmaf(ef, KINC_F_LN2_HI, thi);
   const float s = hi + z;
   const float err = (hi - s) + z;
   const float lo = fmaf(ef, KINC_F_LN2_LO, tlo) + err;
   return s + fmaf(z2, q, lo);
}

/* 16 bytes of shared memory into v, on the lanes with `act` only (the others keep v and take no part in
 * the access); a predicated instruction, so it stays inside straight-line code */
__device__ __forceinline__ void gp_lds4(float4& v, uint32_t addr, int act)
{
   asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %5, 0;\n\t@p ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
                : "+f"(v.x), "+f"(v.y), "+f"(v.z), "+f"(v.w)
                : "r"(addr), "r"(act) : "memory");
}

/* acc + the first cnt (1..GP_CHUNK) floats at a 16-byte aligned shared-memory address, in order; 64 floats
 * may be read there on every lane */
__device__ __forceinline__ float gp_ordered_tail(uint32_t from, int cnt, float acc)
{
   auto load = [&](float4 (&q)[4], uint32_t at) {
#pragma unroll
      for ( int g = 0; g < 4; ++g )
         asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                      : "=f"(q[g].x), "=f"(q[g].y), "=f"(q[g].z), "=f"(q[g].w)
                      : "r"(at + 16 * g) : "memory");
   };
   auto add16 = [&](const float4 (&q)[4]) {
#pragma unroll
      for ( int g = 0; g < 4; ++g )
      {
         acc += q[g].x;
         acc += q[g].y;
         acc += q[g].z;
         acc += q[g].w;
      }
   };
   /* 16 floats ahead of the additions */
   float4 v[4], w[4];
   load(v, from);
   load(w, from + 64);
   if ( cnt >= 32 )
   {
      add16(v);
      load(v, from + 128);
      add16(w);
      load(w, from + 192);
      cnt -= 32;
   }
   if ( cnt >= 16 )
   {
      add16(v);
#pragma unroll
      for ( int g = 0; g < 4; ++g ) v[g] = w[g];
      if ( cnt == 32 )
      {
         add16(v);
         return acc;
      }
      cnt -= 16;
   }
   auto add = [&](float x, int i) { acc = i < cnt ? acc + x : acc; };
#pragma unroll
   for ( int g = 0; g < 4; ++g )
   {
      add(v[g].x, 4 * g);
      add(v[g].y, 4 * g + 1);
      add(v[g].z, 4 * g + 2);
      add(v[g].w, 4 * g + 3);
   }
   return acc;
}

/* log-density of two samples under one component (calcLogMvNorm, the operations of log_mvn) */
__device__ __forceinline__ F2 gp_density(F2 x0, F2 x1, F2 m0, F2 m1, F2 a, F2 b, F2 c, F2 nrm, F2 z)
{
   const F2 xm0 = x0 - m0;
   const F2 xm1 = x1 - m1;
   const F2 b0 = mulz(a, xm0, z) + mulz(b, xm1, z);
   const F2 b1 = mulz(b, xm0, z) + mulz(c, xm1, z);
   const F2 dot = mulz(xm0, b0, z) + mulz(xm1, b1, z);
   /* nrm - 0.5 * dot: halving is exact unless dot is subnormal, which nrm absorbs */
   return fma2(f2(-0.5f), dot, nrm);
}

/*
 * E step for finite parameters and samples: log p(x) of every sample, log(gamma/pi) (into vg), and
 * each component's largest log(gamma/pi) (into par).  KEEP: the parameters stay in registers, 14 for each
 * component; else they are read again for every chunk.
 */
template <int K, bool G, bool KEEP>
__device__ __forceinline__ void gp_e_step(const GpView& s, const GpLogTable& lt, int lane)
{
   const F2 z = f2(s.nz);
   F2 q[K][7];
   float ga[K], gb[K];
   auto parameters = [&](int k) {
#pragma unroll
      for ( int i = 0; i < 3; ++i )
      {
         const float4 v = *reinterpret_cast<const float4*>(s.par + k * GP_PAR + 4 * i);
         q[k][2 * i] = f2(v.x, v.y);
         q[k][2 * i + 1] = f2(v.z, v.w);
      }
      q[k][6] = gp_ld2(s.par + k * GP_PAR + 12);
   };
#pragma unroll
   for ( int k = 0; k < K; ++k )
   {
      if ( KEEP ) parameters(k);
      ga[k] = -INFINITY;
      gb[k] = -INFINITY;
   }
   const float* in = s.x + 4 * lane;
   float* pv = s.vg + 2 * lane;
   float* pl = s.lpx + 2 * lane;
   float4 xn = *reinterpret_cast<const float4*>(in);
#pragma unroll 1
   for ( int c = 0; c < s.nch; ++c )
   {
      const F2 x0 = f2(xn.x, xn.y), x1 = f2(xn.z, xn.w);
      in += c + 1 < s.nch ? 2 * GP_CHUNK : 0;
      xn = *reinterpret_cast<const float4*>(in);
      F2 lg[K], lp[K];
      float ma = -INFINITY, mb = -INFINITY;
#pragma unroll
      for ( int k = 0; k < K; ++k )
      {
         if ( !KEEP ) parameters(k);
         lg[k] = gp_density(x0, x1, q[k][0], q[k][1], q[k][2], q[k][3], q[k][4], q[k][5], z);
         lp[k] = q[k][6] + lg[k];
         float a, b;
         split(lp[k], a, b);
         ma = fmaxf(ma, a);
         mb = fmaxf(mb, b);
      }
      const F2 mm = f2(ma, mb);
      F2 sum;
#pragma unroll
      for ( int k = 0; k < K; ++k )
      {
         const F2 e = gp_exp_beside_one(lp[k] - mm);
         sum = k == 0 ? e : sum + e;
      }
      float sa, sb;
      split(sum, sa, sb);
      const F2 logpx = mm + f2(gp_log(sa, lt), gp_log(sb, lt));
      gp_st2(pl, logpx);
#pragma unroll
      for ( int k = 0; k < K; ++k )
      {
         const F2 v = lg[k] - logpx;
         gp_stv<G>(pv + k * s.n64, v);
         float a, b;
         split(v, a, b);
         ga[k] = fmaxf(ga[k], a);
         gb[k] = fmaxf(gb[k], b);
      }
      pv += GP_CHUNK;
      pl += GP_CHUNK;
   }
   float mine = 0.f;
#pragma unroll
   for ( int k = 0; k < K; ++k )
   {
      const float m = gp_warp_max(fmaxf(ga[k], gb[k]));
      mine = lane == k ? m : mine;
   }
   if ( lane < K ) gp_st2(s.par + lane * GP_PAR + 14, f2(mine));
   __syncwarp();
}

/* the same for any values (NaN, infinities, weights below e^-1e6) */
__device__ __noinline__ void gp_e_step_any(GpView s, int K, int lane)
{
   for ( int k = 0; k < K; ++k )
   {
      const float* q = s.par + k * GP_PAR;
      for ( int i = lane; i < s.nch * GP_CHUNK; i += 32 )
      {
         const float2 x = gp_x(s, i);
         s.vg[k * s.n64 + i] = log_mvn(x.x, x.y, q[0], q[2], q[4], q[6], q[8], q[10]);
      }
   }
   for ( int i = lane; i < s.nch * GP_CHUNK; i += 32 )
   {
      float m = -INFINITY;
      for ( int k = 0; k < K; ++k ) m = fmaxf(m, s.par[k * GP_PAR + 12] + s.vg[k * s.n64 + i]);
      float sum = 0.0f;
      for ( int k = 0; k < K; ++k ) sum += kinc_expf((s.par[k * GP_PAR + 12] + s.vg[k * s.n64 + i]) - m);
      const float logpx = m + kinc_logf(sum);
      s.lpx[i] = logpx;
      for ( int k = 0; k < K; ++k ) s.vg[k * s.n64 + i] = s.vg[k * s.n64 + i] + (-logpx);
   }
   for ( int k = 0; k < K; ++k )
   {
      float g = -INFINITY;
      for ( int i = lane; i < s.nch * GP_CHUNK; i += 32 ) g = fmaxf(g, s.vg[k * s.n64 + i]);
      for ( int o = 16; o > 0; o >>= 1 ) g = fmaxf(g, __shfl_xor_sync(0xffffffffu, g, o));
      if ( lane == 0 ) gp_st2(s.par + k * GP_PAR + 14, f2(g));
   }
   __syncwarp();
}

/* the term rows of one component: its parameters, and how the three rows are formed from its vg */
template <bool G>
struct GpM1Terms
{
   F2 mg;
   __device__ __forceinline__ void init(const float* par) { mg = gp_ld2(par + 14); }
   __device__ __forceinline__ void store(F2 v, F2 x0, F2 x1, float* pv, float* out, int rows) const
   {
      const F2 e = gp_exp(v - mg);
      const F2 g = gp_exp(v);
      gp_st2(out, e);
      gp_st2(out + rows, g * x0);
      gp_st2(out + 2 * rows, g * x1);
      gp_stv<G>(pv, g);
   }
};

struct GpM2Terms
{
   F2 m0, m1;
   __device__ __forceinline__ void init(const float* par)
   {
      m0 = gp_ld2(par);
      m1 = gp_ld2(par + 2);
   }
   __device__ __forceinline__ void store(F2 g, F2 x0, F2 x1, float*, float* out, int rows) const
   {
      const F2 xm0 = x0 - m0;
      const F2 xm1 = x1 - m1;
      gp_st2(out, g * (xm0 * xm0));
      gp_st2(out + rows, g * (xm0 * xm1));
      gp_st2(out + 2 * rows, g * (xm1 * xm1));
   }
};

/*
 * The terms of chunk after chunk and, interleaved with them, the ordered sums of the chunk before:
 * beside each component's terms a K-th of the earlier chunk's 64 samples are added.  The sums are one
 * chain of dependent additions per row and the terms independent arithmetic, so each hides the
 * other's latency; two sets of rows alternate.  The samples to add beside a component's terms are loaded before
 * those, its vg one component ahead (the stores of one may not be passed by the loads of the next), or
 * from global memory one chunk ahead.  `lik`: this lane sums s.lpx
 * instead of a term row.  Returns this lane's sum.
 */
template <int K, bool G, class Terms>
__device__ __forceinline__ float gp_terms_and_sums(const GpView& s, bool lik, bool act, int lane)
{
   constexpr int BUF = 3 * K * GP_ROW;      /* floats of one chunk's rows */
   constexpr int NG = GP_CHUNK / 4;         /* 16-byte groups of a row */
   constexpr int GM = (NG + K - 1) / K;     /* groups beside one component, at most */
   const float* row = lik ? s.lpx : s.terms + (act ? lane : 0) * GP_ROW;
   /* where the lane's next chunk of sums lies: its row alternates between the two sets, log p(x) moves on */
   uint32_t from = (uint32_t)__cvta_generic_to_shared(row) + (lik ? 0u : (uint32_t)sizeof(float) * BUF);
   const uint32_t first = (uint32_t)__cvta_generic_to_shared(row);
   const int sgn = lik ? 1 : -1;
   const uint32_t move = lik ? (uint32_t)sizeof(float) * GP_CHUNK : first + from;
   /* four copies of `act` that the compiler cannot tell to be equal: loads in a row under one predicate
    * were turned into a branch around them (13 cycles each) */
   const int zero = __float_as_int(s.nz) << 1;
   int flag[4];
#pragma unroll
   for ( int i = 0; i < 4; ++i ) flag[i] = (act ? 1 : 0) + (zero >> i);
   float4 v[GM];
#pragma unroll
   for ( int g = 0; g < GM; ++g ) v[g] = make_float4(0.f, 0.f, 0.f, 0.f);
   float acc = 0.f;
   float* out = s.terms + 2 * lane;
   const float* in = s.x + 4 * lane;
   float* pv = s.vg + 2 * lane;
   int flip = BUF;
   Terms t[K];
#pragma unroll
   for ( int k = 0; k < K; ++k ) t[k].init(s.par + k * GP_PAR);
   F2 val[K], next[K];
#pragma unroll
   for ( int k = 0; k < K && G; ++k ) next[k] = gp_ldv<G>(pv + k * s.n64);
#pragma unroll 1
   for ( int c = 0; c < s.nch; ++c )
   {
      const float4 xq = *reinterpret_cast<const float4*>(in);
      const F2 x0 = f2(xq.x, xq.y), x1 = f2(xq.z, xq.w);
      if ( G )
      {
         const int ahead = c + 1 < s.nch ? GP_CHUNK : 0;
#pragma unroll
         for ( int k = 0; k < K; ++k )
         {
            val[k] = next[k];
            next[k] = gp_ldv<G>(pv + k * s.n64 + ahead);
         }
      }
      auto load = [&](int k) {
#pragma unroll
         for ( int g = NG * k / K; g < NG * (k + 1) / K; ++g )
            gp_lds4(v[g - NG * k / K], from + 16 * g, flag[g & 3]);
      };
      if ( !G ) val[0] = gp_ldv<G>(pv);
      load(0);
#pragma unroll
      for ( int k = 0; k < K; ++k )
      {
         if ( !G && k + 1 < K ) val[k + 1] = gp_ldv<G>(pv + (k + 1) * s.n64);
         t[k].store(val[k], x0, x1, pv + k * s.n64, out + k * GP_ROW, K * GP_ROW);
#pragma unroll
         for ( int g = 0; g < NG * (k + 1) / K - NG * k / K; ++g )
         {
            acc += v[g].x;
            acc += v[g].y;
            acc += v[g].z;
            acc += v[g].w;
         }
         if ( k + 1 < K ) load(k + 1);
      }
      /* the first chunk's sums were of nothing; log p(x) starts over */
      acc = c == 0 ? 0.f : acc;
      from = c == 0 ? first : (uint32_t)(sgn * (int)from) + move;
      out += flip;
      flip = -flip;
      in += 2 * GP_CHUNK;
      pv += GP_CHUNK;
      __syncwarp();
   }
   acc = gp_ordered_tail(from, s.N - (s.nch - 1) * GP_CHUNK, acc);
   __syncwarp();
   return acc;
}

/* M step, pass 1: rows k = sum of exp(v - max), K + k and 2K + k = mean sums, 3K = log-likelihood;
 * lane r returns row r's sum.  vg becomes gamma/pi.  For v <= 70 without NaN. */
template <int K, bool G>
__device__ __forceinline__ float gp_m1_step(const GpView& s, int lane)
{
   return gp_terms_and_sums<K, G, GpM1Terms<G>>(s, lane == 3 * K, lane <= 3 * K, lane);
}

/* the same for any values */
__device__ __noinline__ float gp_m1_step_any(GpView s, int K, int lane)
{
   const bool lik = lane == 3 * K;
   float acc = 0.f;
   for ( int i0 = 0; i0 < s.N; i0 += GP_CHUNK )
   {
      const int cnt = min(GP_CHUNK, s.N - i0);
      for ( int k = 0; k < K; ++k )
      {
         const float mg = s.par[k * GP_PAR + 14];
         for ( int i = lane; i < cnt; i += 32 )
         {
            const float2 x = gp_x(s, i0 + i);
            const float v = s.vg[k * s.n64 + i0 + i];
            const float g = kinc_expf(v);
            s.terms[k * GP_ROW + i] = kinc_expf(v - mg);
            s.terms[(K + k) * GP_ROW + i] = g * x.x;
            s.terms[(2 * K + k) * GP_ROW + i] = g * x.y;
            s.vg[k * s.n64 + i0 + i] = g;
         }
      }
      __syncwarp();
      const float* row = lik ? s.lpx + i0 : s.terms + (lane < 3 * K ? lane : 0) * GP_ROW;
      acc = gp_ordered_tail((uint32_t)__cvta_generic_to_shared(row), cnt, acc);
      __syncwarp();
   }
   return acc;
}

/* M step, pass 2: rows k, K + k, 2K + k = the sums of Sigma's elements 00, 01, 11 around the new means
 * (in par) */
template <int K, bool G>
__device__ __forceinline__ float gp_m2_step(const GpView& s, int lane)
{
   return gp_terms_and_sums<K, G, GpM2Terms>(s, false, lane < 3 * K, lane);
}

/* glibc rand() (or the per-fit LCG) drawn by the warp: lane r < 31 holds word r of the state */
struct GpRng
{
   uint32_t word;
   int head, mode;
   uint64_t lcg;

   __device__ __forceinline__ int32_t next(int lane)
   {
      if ( mode == 0 )
      {
         int h28 = head + 28;
         if ( h28 >= RNG_WORDS ) h28 -= RNG_WORDS;
         const uint32_t v = __shfl_sync(0xffffffffu, word, head) + __shfl_sync(0xffffffffu, word, h28);
         if ( lane == head ) word = v;
         head = head + 1 == RNG_WORDS ? 0 : head + 1;
         return (int32_t)(v >> 1);
      }
      lcg = lcg * 1103515245ull + 12345ull;
      return (int32_t)((uint32_t)(lcg / 65536ull) % 32768u);
   }
};

/* what a fit returns; the work labels are left at the start of lpx */
struct GpFit
{
   bool ok;
   int iters;
   float logL, E;
};

/*
 * GMM::fit with K components for the warp's pair, started from sample `draws` of lane k for component k.  Component k's parameters and their update live on
 * lane k.  The M1 pass that finds the log-likelihood unchanged has already overwritten vg, so the
 * E step is repeated then (its parameters are still in par) to give the label pass what the
 * reference's loggamma array holds.
 */
template <int K, bool G, int WARPS>
__device__ __noinline__ GpFit gp_fit(GpLayout lay, double c2, bool ocl, bool icl, bool xsafe, int draws, int lane)
{
   GpView s = lay.view();
   if ( G ) s.vg = lay.vg_global;
   GpLogTable lt;
   lt.load(lane);
   GpFit out;
   out.ok = false;
   out.iters = 0;
   out.logL = out.E = 0.f;

   /* component kk on lanes kk, K + kk and 2K + kk: the first forms its weight, the others one mean each,
    * and all three one element of the inverse covariance; the lanes beyond repeat component 0 */
   const int role = lane / K < 3 ? lane / K : 3;
   const int kk = role < 3 ? lane % K : 0;
   float* par = s.par + kk * GP_PAR;
   auto publish = [&](int at, float v) { gp_st2(par + at, f2(v)); };
   const float2 start = gp_x(s, __shfl_sync(0xffffffffu, draws, kk));
   float m = role == 1 ? start.x : start.y;
   if ( role == 1 || role == 2 ) publish(2 * role - 2, m);
   float lpi = kinc_logf(1.0f / K), sc = 1.f;
   float s00 = 1.f, s01 = 0.f, s11 = 1.f;

   float prevL = -INFINITY, curL = -INFINITY;
   bool converged = false, safe = false;
   for ( int t = 0;; ++t )
   {
      if ( !converged )
      {
         /* matrixInverse + prepareCovariance (the operations of prepare_cov); the covariances of the
          * last iteration are only checked (at first: the identity) */
         const float t00 = s00 * sc, t01 = s01 * sc, t11 = s11 * sc;
         const float det = t00 * t11 - t01 * t01;
         const bool bad = ocl ? fabsf(det) <= 0.f : det <= 0;
         if ( __any_sync(0xffffffffu, bad) ) return out;
         if ( t == 100 ) break;
         ++out.iters;
         const bool normal = __float_as_uint(det) - 0x00800000u < 0x7f000000u;
         const float logdet = __all_sync(0xffffffffu, normal) ? gp_log(det, lt) : kinc_logf(det);
         const float nrm = (float)(-0.5 * (c2 + (double)logdet));
         const float inv = (role == 0 ? t11 : role == 1 ? -t01 : t00) / det;
         if ( role < 3 ) publish(4 + 2 * role, inv);
         if ( role == 0 )
         {
            publish(10, nrm);
            publish(12, lpi);
         }
         /* with these bounds (and |x| <= 1e8) every log-density is finite: no product exceeds 2e29 */
         const bool bounded = role == 3 || (fabsf(inv) <= 1e12f && (role == 0 ? fabsf(nrm) <= 1e6f && fabsf(lpi) <= 1e6f
                                                                              : fabsf(m) <= 1e8f));
         safe = xsafe && __all_sync(0xffffffffu, bounded);
         __syncwarp();
      }
      if ( safe )
         gp_e_step<K, G, WARPS == GP_WARPS_FEW || K <= 3>(s, lt, lane);
      else
         gp_e_step_any(s, K, lane);
      if ( converged ) break;
      const float mg = par[14];
      /* finite densities: the sums below hold an exp(0) = 1 and are at least that */
      const bool fast = safe && __all_sync(0xffffffffu, mg <= 70.0f);
      float acc = fast ? gp_m1_step<K, G>(s, lane) : gp_m1_step_any(s, K, lane);
      prevL = curL;
      curL = __shfl_sync(0xffffffffu, acc, 3 * K);
      if ( fabsf(curL - prevL) < 1e-8f )
      {
         converged = true;
         continue;
      }

      /* the new weights and means */
      auto log_of = [&](float x) { return fast ? gp_log(x, lt) : kinc_logf(x); };
      const float logGamma = mg + log_of(__shfl_sync(0xffffffffu, acc, kk));
      const float arg = lpi + logGamma;
      float mx = -INFINITY;
#pragma unroll
      for ( int k = 0; k < K; ++k ) mx = fmaxf(mx, __shfl_sync(0xffffffffu, arg, k));
      const float ex = kinc_expf(arg - mx);
      float sum = 0.f;
#pragma unroll
      for ( int k = 0; k < K; ++k ) sum += __shfl_sync(0xffffffffu, ex, k);
      const float lgs = mx + log_of(sum);
      lpi += logGamma - lgs;
      sc = 1.0f / kinc_expf(logGamma);
      m = acc * sc;
      if ( role == 1 || role == 2 ) publish(2 * role - 2, m);
      __syncwarp();

      acc = gp_m2_step<K, G>(s, lane);
      s00 = __shfl_sync(0xffffffffu, acc, kk);
      s01 = __shfl_sync(0xffffffffu, acc, K + kk);
      s11 = __shfl_sync(0xffffffffu, acc, 2 * K + kk);
   }

   /* ---- calcLabels + calcEntropy: log(gamma/pi) of the last E step if EM converged, gamma/pi if it
    * ran out of iterations */
   float E = 0.f;
   int8_t* wl = reinterpret_cast<int8_t*>(s.lpx);
   for ( int c = 0; c < s.nch; ++c )
   {
      const int i = c * GP_CHUNK + 2 * lane;
      int ka = -1, kb = -1;
      float ga = -INFINITY, gb = -INFINITY;
#pragma unroll
      for ( int k = 0; k < K; ++k )
      {
         float a, b;
         split(gp_ldv<G>(s.vg + k * s.n64 + i), a, b);
         if ( ga < a )
         {
            ka = k;
            ga = a;
         }
         if ( gb < b )
         {
            kb = k;
            gb = b;
         }
      }
      *reinterpret_cast<char2*>(wl + i) = make_char2((char)ka, (char)kb);
      if ( icl )
      {
         const float nan = __int_as_float(0x7fc00000);
         gp_st2(s.terms + 2 * lane, f2(ka >= 0 ? kinc_logf(ga) : nan, kb >= 0 ? kinc_logf(gb) : nan));
         __syncwarp();
         E = gp_ordered_tail((uint32_t)__cvta_generic_to_shared(s.terms), min(GP_CHUNK, s.N - c * GP_CHUNK), E);
         __syncwarp();
      }
   }
   __syncwarp();
   out.ok = true;
   out.logL = curL;
   out.E = E;
   return out;
}

/* fetchPair into the pair's arrays: returns N, fills x up to whole chunks by repeating the first
 * sample (so no maximum changes), and tells whether every |value| <= 1e8 */
__device__ inline int gp_fetch(const DevParams& P, const DevData& D, int32_t x, int32_t y, const GpView& s,
                               int8_t* lbl, int lane, bool& xsafe)
{
   bool fine = true;
   const int n = pair_fetch(P, D, x, y, lbl, lane, [&](int at, float v0, float v1) {
      if ( at >= s.n64 ) return;
      float* q = s.x + (at >> 1) * 4 + (at & 1);
      q[0] = v0;
      q[2] = v1;
      fine = fine && fabsf(v0) <= 1e8f && fabsf(v1) <= 1e8f;
   });
   if ( n > 0 && n <= s.n64 )
   {
      const float2 first = gp_x(s, 0);
      const int end = (n + GP_CHUNK - 1) / GP_CHUNK * GP_CHUNK;
      for ( int i = n + lane; i < end; i += 32 )
      {
         float* q = s.x + (i >> 1) * 4 + (i & 1);
         q[0] = first.x;
         q[2] = first.y;
      }
   }
   xsafe = __all_sync(0xffffffffu, fine);
   __syncwarp();
   return n;
}

/* the CTA's active warps wait for one another */
__device__ __forceinline__ void gp_cta_sync(int warps)
{
   asm volatile("bar.sync 1, %0;" ::"r"(warps * 32) : "memory");
}

/*
 * One CTA per SM; its shared memory is cut into as many pair slots as the block's largest usable
 * count allows (the pairs come ordered by count), one warp per slot.  A CTA takes a group of
 * consecutive pairs, one per warp, and its warps begin the fit of each K together: they then run the
 * same code, which does not fit the instruction caches for all K at once (nearly all fits run the
 * full 100 iterations, so little is waited for).  When there are fewer pairs than slots, the groups
 * are smaller and every SM gets some.
 */
template <int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 1)
k_gmm_pairs(DevParams P, DevData D, DevScratch W, DevBlock B, int smem_floats, int sort_rows, int n_cap)
{
   extern __shared__ __align__(16) float gp_shared[];
   const int lane = threadIdx.x & 31;
   const int warp = threadIdx.x >> 5;
   const int n_most = B.order ? min(n_cap, B.N[B.start + B.order[0] - B.lo]) : n_cap;
   /* log(gamma/pi) in shared memory where that still leaves enough pairs to an SM */
   const bool in_global = smem_floats / gp_slot_floats(max(n_most, 1), P.max_k, sort_rows, false) < gp_shared_pairs(WARPS);
   const int slot_floats = gp_slot_floats(max(n_most, 1), P.max_k, sort_rows, in_global);
   const int64_t per_cta = (B.size + gridDim.x - 1) / gridDim.x;
   const int slots = min(WARPS, smem_floats / slot_floats);
   const int warps = per_cta < slots ? (int)per_cta : slots;
   if ( warp >= warps ) return;
   const int64_t groups = (B.size + warps - 1) / warps;
   __shared__ unsigned long long next_group;

   GpLayout lay;
   lay.n64 = (max(n_most, 1) + GP_CHUNK - 1) / GP_CHUNK * GP_CHUNK;
   lay.x = warp * slot_floats;
   lay.par = lay.x + 2 * lay.n64;
   lay.terms = lay.par + GP_KMAX * GP_PAR;
   lay.vg = lay.terms + 2 * 3 * P.max_k * GP_ROW;
   const int lpx0 = lay.vg + (in_global ? 0 : P.max_k * lay.n64);
   lay.vg_global = W.gam + ((size_t)blockIdx.x * GP_WARPS + warp) * (size_t)gp_global_floats(n_cap, P.max_k);
   lay.lpx = lpx0;
   lay.nz = P.neg_zero;
   lay.N = lay.nch = 0;

   for ( int64_t group = blockIdx.x; group < groups; )
   {
      const int64_t q = group * warps + warp;
      const bool live = q < B.size;
      const int64_t p = B.start + (!live ? 0 : B.order ? B.order[q] : q);
      int32_t x, y;
      pair_xy(p, x, y);
      int8_t* lbl = B.outLabels ? B.outLabels + (p - B.start) * (int64_t)P.S
                                : W.lbl + ((size_t)blockIdx.x * GP_WARPS + warp) * (size_t)P.S;
      GpView s = lay.view();
      GpRng rng;
      bool fits = false, xsafe = false;
      int n = 0, K = 0;
      if ( live )
      {
         n = gp_fetch(P, D, x, y, s, lbl, lane, xsafe);
         if ( n != B.N[p - B.lo] || n > s.n64 )
         {
            if ( lane == 0 ) atomicCAS(B.status, ST_OK, ST_BAD_RANK);
            n = 0;
         }
         s.N = n;
         s.nch = (n + GP_CHUNK - 1) / GP_CHUNK;
         if ( P.pre_out )
         {
            pair_mark_outliers(GpSamples { s }, n, s.work, 0, lbl, 0, -7, lane);
            pair_mark_outliers(GpSamples { s }, n, s.work, 1, lbl, 0, -7, lane);
         }
         fits = n >= P.min_samples;
         rng.mode = P.rand_mode;
         rng.head = 0;
         rng.lcg = 1;
         rng.word = fits && rng.mode == 0
                       ? warp_rng_state(D, B.qpos[p - B.start] * (uint64_t)P.draws_per_pair, lane) : 0;
      }
      float bestValue = INFINITY;
      unsigned long long units = 0;
      for ( int k = P.min_k; k <= P.max_k; ++k )
      {
         gp_cta_sync(warps);
         if ( !fits ) continue;
         /* the means start at k samples drawn from rand(), the draw of component j on lane j */
         if ( rng.mode == 1 ) rng.lcg = 1;
         int draw = 0;
         for ( int j = 0; j < k; ++j )
         {
            const int ii = rng.next(lane) % n;
            if ( lane == j ) draw = ii;
         }
         GpLayout l = lay;
         l.N = n;
         l.nch = s.nch;
         /* log p(x) is summed beside 3k term rows: start it 4 banks after the last of them */
         l.lpx = lpx0 + ((12 * k - (lpx0 - lay.terms)) & 31);
         GpFit f;
         const bool ocl = P.rand_mode == 1, icl = P.criterion == 1;
         auto fit = [&](auto g) {
            constexpr bool G = decltype(g)::value;
            switch ( k )
            {
            case 1: return gp_fit<1, G, WARPS>(l, P.c2, ocl, icl, xsafe, draw, lane);
            case 2: return gp_fit<2, G, WARPS>(l, P.c2, ocl, icl, xsafe, draw, lane);
            case 3: return gp_fit<3, G, WARPS>(l, P.c2, ocl, icl, xsafe, draw, lane);
            case 4: return gp_fit<4, G, WARPS>(l, P.c2, ocl, icl, xsafe, draw, lane);
            default: return gp_fit<5, G, WARPS>(l, P.c2, ocl, icl, xsafe, draw, lane);
            }
         };
         f = in_global ? fit(std::true_type()) : fit(std::false_type());
         const int8_t* wl = reinterpret_cast<const int8_t*>(gp_shared + l.lpx);
         units += (unsigned long long)f.iters * n * k;
         if ( !f.ok ) continue;
         const float value = ocl ? criterion_value<true>(P, D, k, f.logL, n, f.E)
                                 : criterion_value<false>(P, D, k, f.logL, n, f.E);
         if ( value < bestValue )
         {
            K = k;
            bestValue = value;
            for ( int i0 = 0, j = 0; i0 < n; i0 += 32 )
            {
               const int i = i0 + lane;
               const bool in = i < n && lbl[i] >= 0;
               const unsigned bal = __ballot_sync(0xffffffffu, in);
               if ( in ) lbl[i] = wl[j + __popc(bal & lanemask_lt())];
               j += __popc(bal);
            }
            __syncwarp();
         }
      }

      if ( live )
      {
         if ( fits && lane == 0 && B.work )
         {
            atomicAdd(&B.work[0], units);
            atomicAdd(&B.work[1], (unsigned long long)(P.max_k - P.min_k + 1));
         }
         pair_finish(P, D, B, GpSamples { s }, s.work, lbl, p, n, K, lane);
      }

      gp_cta_sync(warps);
      if ( threadIdx.x == 0 ) next_group = atomicAdd(B.tiles, 1ull) + gridDim.x;
      gp_cta_sync(warps);
      group = (int64_t)next_group;
   }
}

} /* namespace kinc */
