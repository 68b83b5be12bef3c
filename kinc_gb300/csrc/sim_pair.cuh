/*
 * sim_pair.cuh -- what a warp does with one pair before and after its fits,
 * for the kernels that give a warp whole pairs (sim_gmm_pair.cuh,
 * sim_kmeans_pairs.cuh).  The pair's packed samples are read through `at(i)`,
 * labels are one byte per sample position.
 */
#pragma once

#include "sim_kernel.cuh"

namespace kinc {

/* fetchPair: labels by sample position, put(i, x, y) for the i-th usable sample; returns their number */
template <class Put>
__device__ __forceinline__ int pair_fetch(const DevParams& P, const DevData& D, int32_t x, int32_t y, int8_t* lbl, int lane,
                                          Put put)
{
   const float* g1 = D.gem + (size_t)x * P.S;
   const float* g2 = D.gem + (size_t)y * P.S;
   constexpr int CH = 4;            /* 32-sample chunks whose loads are in flight together */
   int n = 0;
   for ( int base = 0; base < P.S; base += CH * 32 )
   {
      float v1[CH], v2[CH];
#pragma unroll
      for ( int u = 0; u < CH; ++u )
      {
         const int i = base + u * 32 + lane;
         v1[u] = i < P.S ? __ldg(g1 + i) : 0.f;
         v2[u] = i < P.S ? __ldg(g2 + i) : 0.f;
      }
#pragma unroll
      for ( int u = 0; u < CH; ++u )
      {
         const int i = base + u * 32 + lane;
         bool use = false;
         if ( i < P.S )
         {
            const bool nanb = isnan(v1[u]) || isnan(v2[u]);
            const bool low = v1[u] < P.min_expr || v2[u] < P.min_expr;
            lbl[i] = nanb ? (int8_t)-9 : (low ? (int8_t)-6 : (int8_t)0);
            use = !nanb && !low;
         }
         const unsigned bal = __ballot_sync(0xffffffffu, use);
         if ( use ) put(n + __popc(bal & lanemask_lt()), v1[u], v2[u]);
         n += __popc(bal);
      }
   }
   __syncwarp();
   return n;
}

/* warp_bitonic with the pairs of a stage indexed by shifts instead of divisions: K-means k <= 3 of 100 samples 3.05 ->
 * 2.97 ms here.  (The tile kernel keeps the divisions; with shifts Spearman in the allocation-free call, 32,768 pairs,
 * took 4.98 instead of 4.73 ms at 300 samples and 73.7 instead of 68.3 ms at 1,000.) */
__device__ inline void pair_bitonic(int size, float* key, float* extra, int lane)
{
   const int bsize = size / 2;
   for ( int half = 1; half < size; half *= 2 )
   {
      for ( int t = half; t >= 1; t >>= 1 )
      {
         for ( int i = lane; i < bsize; i += 32 )
         {
            /* a = i / t * 2t + i % t; powers of two, so no division */
            const bool desc = (i & half) != 0;
            const int a = 2 * i - (i & (t - 1));
            const int b = a + t;
            const float ka = key[a];
            const float kb = key[b];
            if ( (ka > kb && !desc) || (ka < kb && desc) )
            {
               key[a] = kb;
               key[b] = ka;
               if ( extra )
               {
                  const float ea = extra[a];
                  extra[a] = extra[b];
                  extra[b] = ea;
               }
            }
         }
         __syncwarp();
      }
   }
}

/* Clustering::markOutliers (as warp_mark_outliers) */
template <class X>
__device__ inline void pair_mark_outliers(X at, int N, float* buf, int col, int8_t* lbl, int8_t cluster, int8_t marker,
                                                int lane)
{
   int n = 0;
   for ( int base = 0; base < N; base += 32 )
   {
      const int i = base + lane;
      bool sel = false;
      if ( i < N )
      {
         const int8_t l = lbl[i];
         sel = l == cluster || l == marker;
      }
      const unsigned bal = __ballot_sync(0xffffffffu, sel);
      if ( sel )
      {
         const float2 xv = at(i);
         buf[n + __popc(bal & lanemask_lt())] = col == 0 ? xv.x : xv.y;
      }
      n += __popc(bal);
   }
   if ( n == 0 )
   {
      __syncwarp();
      return;
   }
   const int np2 = next_pow2(n);
   for ( int i = n + lane; i < np2; i += 32 ) buf[i] = __int_as_float(0x7f800000);
   __syncwarp();
   pair_bitonic(np2, buf, nullptr, lane);
   const float Q1 = buf[n * 1 / 4];
   const float Q3 = buf[n * 3 / 4];
   const float T_min = Q1 - 1.5f * (Q3 - Q1);
   const float T_max = Q3 + 1.5f * (Q3 - Q1);
   for ( int i = lane; i < N; i += 32 )
   {
      if ( lbl[i] == cluster )
      {
         const float2 xv = at(i);
         const float v = col == 0 ? xv.x : xv.y;
         if ( v < T_min || T_max < v ) lbl[i] = marker;
      }
   }
   __syncwarp();
}

/* the closing formula of Spearman::computeCluster (pairwise_spearman.cpp:73-82): the sum of squared rank
 * differences and n(n^2 - 1) are ints */
__device__ __forceinline__ float spearman_value(uint32_t diff, int n)
{
   const int32_t denom = (int32_t)((uint32_t)n * ((uint32_t)n * (uint32_t)n - 1u));
   return (float)(1.0 - 6.0 * (double)(int32_t)diff / (double)denom);
}

/* Spearman of n points by the reference's sorting network (sx, sy: room for next_pow2(n) each); the ranks by x
 * take the place of the sorted x */
__device__ inline float spearman_sorted(float* sx, float* sy, int n, int lane)
{
   float* sr = sx;
   const int np2 = next_pow2(n);
   for ( int i = n + lane; i < np2; i += 32 )
   {
      sx[i] = __int_as_float(0x7f800000);
      sy[i] = __int_as_float(0x7f800000);
   }
   __syncwarp();
   pair_bitonic(np2, sx, sy, lane);
   for ( int i = lane; i < np2; i += 32 ) sr[i] = i < n ? (float)(i + 1) : 0.f;
   __syncwarp();
   pair_bitonic(np2, sy, sr, lane);
   uint32_t diff = 0;
   for ( int i = lane; i < n; i += 32 )
   {
      const int tmp = (int)((float)(i + 1) - sr[i]);
      diff += (uint32_t)(tmp * tmp);
   }
   diff = __reduce_add_sync(0xffffffffu, diff);
   __syncwarp();
   return spearman_value(diff, n);
}

/* the same for the samples of two rows that `mask` has (buf: room for two sorts of S) */
__device__ inline float spearman_network(const float* g1, const float* g2, int S, const uint32_t* mask, float* buf, int lane)
{
   float* sx = buf;
   float* sy = buf + next_pow2(S);
   int n = 0;
   for ( int base = 0; base < S; base += 32 )
   {
      const uint32_t m = mask[base >> 5];
      const int at = n + __popc(m & lanemask_lt());
      if ( (m >> lane) & 1u )
      {
         sx[at] = g1[base + lane];
         sy[at] = g2[base + lane];
      }
      n += __popc(m);
   }
   __syncwarp();
   return spearman_sorted(sx, sy, n, lane);
}

/* Spearman::computeCluster (as warp_spearman) */
template <class X>
__device__ inline float pair_spearman(const DevParams& P, const DevData& D, X at, int N, float* buf,
                                            const int8_t* lbl, int32_t x, int32_t y, int8_t k, int lane)
{
   const int p2 = next_pow2(N);
   float* sx = buf;
   float* sy = sx + p2;
   const float* g1 = D.gem + (size_t)x * P.S;
   const float* g2 = D.gem + (size_t)y * P.S;
   int n = 0;
   int jw = 0;
   for ( int base = 0; base < P.S; base += 32 )
   {
      const int i = base + lane;
      const int8_t l = i < P.S ? lbl[i] : (int8_t)-1;
      const bool incl = l == k;
      const unsigned bn = __ballot_sync(0xffffffffu, l >= 0);
      const unsigned bi = __ballot_sync(0xffffffffu, incl);
      if ( incl )
      {
         const int slot = n + __popc(bi & lanemask_lt());
         const float2 v = P.semantics == 0 ? at(jw + __popc(bn & lanemask_lt())) : make_float2(g1[i], g2[i]);
         sx[slot] = v.x;
         sy[slot] = v.y;
      }
      n += __popc(bi);
      jw += __popc(bn);
   }
   if ( n < P.min_samples )
   {
      __syncwarp();
      return __int_as_float(0x7fc00000);
   }
   return spearman_sorted(sx, sy, n, lane);
}

/* Pearson::computeCluster (as lane_pearson) of every cluster k < K <= 5: lane 5k + q sums the q-th of
 * cluster k's five sums, in sample position order; lane k returns cluster k's correlation */
template <class X>
__device__ inline float pair_pearson(const DevParams& P, const DevData& D, const DevBlock& B, X at, int N,
                                           const int8_t* lbl, int64_t p, int32_t x, int32_t y, int lane)
{
   const int k = lane / 5, q = lane % 5;
   float acc = 0.f;
   int n = 0;
   /* the points of up to 32 consecutive positions, one per lane, added in order */
   auto add = [&](float vx, float vy, int l, int cnt) {
      for ( int j = 0; j < cnt; ++j )
      {
         const float ax = __shfl_sync(0xffffffffu, vx, j);
         const float ay = __shfl_sync(0xffffffffu, vy, j);
         const int al = __shfl_sync(0xffffffffu, l, j);
         const float a = q == 1 || q == 3 ? ay : ax;
         const float b = q < 2 ? 1.0f : q == 2 ? ax : ay;
         if ( al == k )
         {
            acc += a * b;
            ++n;
         }
      }
   };
   if ( P.semantics == 0 )
   {
      for ( int base = 0; base < N; base += 32 )
      {
         const int i = base + lane;
         const float2 v = i < N ? at(i) : make_float2(0.f, 0.f);
         add(v.x, v.y, i < N ? lbl[i] : -1, min(32, N - base));
      }
      /* positions i >= N: what the last earlier pair of the work block with more than i usable
       * samples left there (links point strictly backwards, as in lane_pearson) */
      const int32_t self = (int32_t)(p - B.lo);
      for ( int base = N; base < P.S; base += 32 )
      {
         const int i = base + lane;
         const int l = i < P.S ? lbl[i] : -1;
         float2 v = make_float2(0.f, 0.f);
         if ( l >= 0 )
         {
            int32_t c = B.pg[self];
            if ( c >= self ) c = -1;
            while ( c >= 0 && B.N[c] <= i )
            {
               const int32_t nxt = B.pg[c];
               c = nxt < c ? nxt : -1;
            }
            PackedCursor cur;
            if ( c >= 0 ) v = cur.at(P, D, B.lo + c, i);
         }
         __syncwarp();
         add(v.x, v.y, l, min(32, P.S - base));
      }
   }
   else
   {
      const float* g1 = D.gem + (size_t)x * P.S;
      const float* g2 = D.gem + (size_t)y * P.S;
      for ( int base = 0; base < P.S; base += 32 )
      {
         const int i = base + lane;
         const bool in = i < P.S;
         add(in ? g1[i] : 0.f, in ? g2[i] : 0.f, in ? lbl[i] : -1, min(32, P.S - base));
      }
   }
   const int from = lane < 5 ? 5 * lane : 0;
   const float sx = __shfl_sync(0xffffffffu, acc, from), sy = __shfl_sync(0xffffffffu, acc, from + 1);
   const float sxx = __shfl_sync(0xffffffffu, acc, from + 2), syy = __shfl_sync(0xffffffffu, acc, from + 3);
   const float sxy = __shfl_sync(0xffffffffu, acc, from + 4);
   return pearson_value(P, __shfl_sync(0xffffffffu, n, from), sx, sy, sxx, syy, sxy);
}

/* the pair's post-clustering outliers, correlations and K (buf: room for the outlier and Spearman sorts) */
template <class X>
__device__ __forceinline__ void pair_finish(const DevParams& P, const DevData& D, const DevBlock& B, X at, float* buf,
                                            int8_t* lbl, int64_t p, int N, int K, int lane)
{
   int32_t x, y;
   pair_xy(p, x, y);
   if ( P.post_out && K > 1 )
   {
      for ( int k = 0; k < K; ++k )
      {
         pair_mark_outliers(at, N, buf, 0, lbl, (int8_t)k, -8, lane);
         pair_mark_outliers(at, N, buf, 1, lbl, (int8_t)k, -8, lane);
      }
   }
   const int nc = P.ncorr;
   float* row = B.outCorr ? B.outCorr + (p - B.start) * P.max_k * nc : nullptr;
   const float nan = __int_as_float(0x7fc00000);
   if ( P.corr != 1 && row )
   {
      const float r = K > 0 ? pair_pearson(P, D, B, at, N, lbl, p, x, y, lane) : nan;
      if ( lane < P.max_k ) row[lane * nc] = lane < K ? r : nan;
   }
   if ( P.corr != 0 && row )
   {
      for ( int k = 0; k < P.max_k; ++k )
      {
         const float r = k < K ? pair_spearman(P, D, at, N, buf, lbl, x, y, (int8_t)k, lane) : nan;
         if ( lane == 0 ) row[k * nc + (P.corr == 2 ? 1 : 0)] = r;
      }
   }
   if ( lane == 0 && B.outK ) B.outK[p - B.start] = (int8_t)K;
   __syncwarp();
}

} /* namespace kinc */
