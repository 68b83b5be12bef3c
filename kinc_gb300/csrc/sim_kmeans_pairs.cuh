/*
 * sim_kmeans_pairs.cuh -- K-means clustering (up to KT = 3 or 5 clusters):
 * a warp's lanes iterate the runs of a stream of pairs.
 *
 * KMeans::fit (src/core/pairwise_kmeans.cpp:12-99) runs 10 initialisations
 * per cluster count K, each up to 300 Lloyd iterations until no label changes,
 * and keeps the run with the largest log-likelihood; Clustering::compute
 * (src/core/pairwise_clustering.cpp:23-103) does that for K = minclus..maxclus
 * and keeps the K with the best criterion.  The runs of one pair depend on one
 * another only through the rand() stream, whose positions are known in
 * advance, so they are independent tasks.  A warp keeps up to KM_COLS pairs
 * open; a lane whose run has converged takes the next run of any open pair,
 * and when those are all taken the warp opens the next pair of the queue.  A
 * pair whose last run has ended is closed by the whole warp: the runs'
 * log-likelihoods (one lane each), the choice of initialisation and K, the
 * labels, outliers and correlations.  So the slowest run of a pair delays that
 * pair and no other, and few pairs are needed to keep every lane busy.
 *
 * A Lloyd iteration reads each sample once, assigns it by squared distances
 * (km_label) and adds it to its cluster's sums, in sample order; labels are not
 * kept (a run has converged when means and counts repeat).  Every value is
 * computed by the reference's operation sequence, so the results are those of
 * the serial code.
 *
 * Against a pool per 32-pair tile (the earlier form: a warp waited for the
 * tile's slowest run, kept every iteration's labels and took an IEEE square
 * root per distance), earlier -> now: 65,536 pairs of 4,000 samples (0-60 %
 * missing, k <= 3, BIC, Pearson) 1,060 -> 146 ms, 262,144 such pairs 1,804 ->
 * 536 ms, 22,155 pairs of 333 samples (k <= 5, ICL, Spearman) 107 -> 6.2 ms.
 * Issue slots bound it: 0.72 of them used, 25 warp instructions per 32 (sample,
 * cluster, iteration) units, two thirds of them the sweeps'.  KM_COLS 4, 8, 16:
 * 144, 146, 156 ms; two CTAs per SM at 64 registers 165 ms.
 */
#pragma once

#include "sim_pair.cuh"

#include <type_traits>

namespace kinc {

/* offset of run (K, init) in a pair's draws */
__device__ __forceinline__ int km_draw_offset(int kmin, int K, int init)
{
   return 10 * ((K - 1) * K / 2 - (kmin - 1) * kmin / 2) + init * K;
}

/* a pair's run t: K descending (the longest runs first), 10 initialisations each */
__device__ __forceinline__ int km_run_k(int kmax, int t)
{
   return kmax - t / 10;
}

/* label of x under means (m0, m1)[0..K): the reference's first-minimum rule */
template <int KT>
__device__ __forceinline__ int km_assign(float x0, float x1, const float* m0, const float* m1, int K, float& min_d)
{
   int min_k = -1;
   min_d = 0.f;
#pragma unroll
   for ( int k = 0; k < KT; ++k )
   {
      if ( k >= K ) continue;
      const float d = diff_norm(x0, x1, m0[k], m1[k]);
      if ( min_k == -1 || d < min_d )
      {
         min_k = k;
         min_d = d;
      }
   }
   return min_k;
}

/* vectorDiffNorm's sum of squares, before the root; z: -0 (kinc_f2.h, mulz) */
__device__ __forceinline__ float km_square(F2 x, F2 mu, F2 z)
{
   const F2 d = x - mu;
   float a, b;
   split(mulz(d, d, z), a, b);
   return a + b;
}

/*
 * The same label from the squared distances.  The rounded square root never decreases, so a squared
 * distance that is not smaller does not win, and one that is smaller by more than two parts in 2^22 wins
 * (two floats with the same rounded root differ by less; 2^-20 is taken); in between -- and where the
 * squares are too small for that to hold -- `near` is set and the roots decide.  A NaN mean (an empty
 * cluster's, or the place of a component that the run does not have) never wins over another.
 */
template <int KM>
__device__ __forceinline__ int km_label(F2 x, const F2 (&mu)[KM], F2 z, bool& near)
{
   int l = 0;
   float best = km_square(x, mu[0], z);
#pragma unroll
   for ( int k = 1; k < KM; ++k )
   {
      const float q = km_square(x, mu[k], z);
      const bool less = q < best;
      near = near || (less && !(q < fmaf(best, 0.99999904632568359375f, -1e-35f)));
      best = less ? q : best;
      l = less ? k : l;
   }
   return l;
}

template <int KM>
__device__ __noinline__ int km_label_by_roots(F2 x, const F2 (&mu)[KM])
{
   float m0[KM], m1[KM], d;
#pragma unroll
   for ( int k = 0; k < KM; ++k ) split(mu[k], m0[k], m1[k]);
   return km_assign<KM>(lo(x), hi(x), m0, m1, KM, d);
}

/* x into cluster l's sums: for every k one predicated addition (as a branch each cost 13 cycles) */
template <int KM>
__device__ __forceinline__ void km_add(F2 x, int l, F2 (&s)[KM], int (&n)[KM])
{
#pragma unroll
   for ( int k = 0; k < KM; ++k )
      asm("{\n\t.reg .pred p;\n\tsetp.eq.s32 p, %2, %4;\n\t@p add.rn.f32x2 %0, %0, %3;\n\t@p add.s32 %1, %1, 1;\n\t}"
          : "+l"(s[k].v), "+r"(n[k])
          : "r"(l), "l"(x.v), "r"(k));
}

/*
 * The open pairs' samples on their way through shared memory: a warp's lanes are all at the same sample,
 * so one row (that sample of the KM_COLS open pairs) serves every lane, whichever pair its run belongs
 * to.  Stages of KM_STAGE rows are copied KM_DEPTH - 1 stages ahead of their use.
 */
struct KmStream
{
   const float2* X;             /* [S][KM_COLS] */
   uint32_t ring;               /* shared-memory address */
   int S, lane;                 /* rows of X */

   /* starts the copy of stage t; every lane calls it */
   __device__ __forceinline__ void start(int t) const
   {
      constexpr int PER_ROW = KM_COLS / 2;                 /* 16-byte pieces of a row */
      const uint32_t to = ring + (uint32_t)(t % KM_DEPTH) * (KM_STAGE * KM_COLS * 8);
#pragma unroll
      for ( int i = lane; i < KM_STAGE * PER_ROW; i += 32 )
      {
         const int row = min(t * KM_STAGE + i / PER_ROW, S - 1);
         const float2* from = X + row * KM_COLS + (i % PER_ROW) * 2;
         asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + 16 * i), "l"(from) : "memory");
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
   }
   /* an empty group in a stage's place, so the count of groups in flight stays the same */
   __device__ __forceinline__ void skip() const { asm volatile("cp.async.commit_group;" ::: "memory"); }
   /* stage t has arrived for every lane, and the stage before it has been used by every lane */
   __device__ __forceinline__ void wait() const
   {
      asm volatile("cp.async.wait_group %0;" ::"n"(KM_DEPTH - 2) : "memory");
      __syncwarp();
   }
};

/*
 * One Lloyd iteration of a lane's run: every sample of its column j is assigned and
 * added to its cluster's sums, in sample order.  `all`: samples every active lane has; `most`: samples of
 * the longest (a lane adds its first `lim`).
 */
template <int KM>
__device__ __forceinline__ void km_sweep(const KmStream& x, int j, int lim, int all, int most, const F2 (&mu)[KM], F2 z,
                                         F2 (&s)[KM], int (&n)[KM])
{
   constexpr int U = 4;
#pragma unroll
   for ( int k = 0; k < KM; ++k )
   {
      s[k] = f2(0.f);
      n[k] = 0;
   }
   const int stages = (most + KM_STAGE - 1) / KM_STAGE;
   __syncwarp();                                           /* the ring's last readers are done */
#pragma unroll
   for ( int t = 0; t < KM_DEPTH - 1; ++t )
   {
      if ( t < stages )
         x.start(t);
      else
         x.skip();
   }
   constexpr uint32_t row = KM_COLS * 8;
#pragma unroll 1
   for ( int t = 0; t < stages; ++t )
   {
      x.wait();
      if ( t + KM_DEPTH - 1 < stages )
         x.start(t + KM_DEPTH - 1);
      else
         x.skip();
      uint32_t at = x.ring + (uint32_t)(t % KM_DEPTH) * (KM_STAGE * row) + 8 * j;
#pragma unroll 1
      for ( int i = t * KM_STAGE; i < min(t * KM_STAGE + KM_STAGE, most); i += U )
      {
         F2 xv[U];
         int l[U];
#pragma unroll
         for ( int u = 0; u < U; ++u )
         {
            asm volatile("ld.shared.b64 %0, [%1];" : "=l"(xv[u].v) : "r"(at + u * row) : "memory");
         }
         at += U * row;
         bool near = false;
#pragma unroll
         for ( int u = 0; u < U; ++u ) l[u] = km_label<KM>(xv[u], mu, z, near);
         if ( near )
         {
#pragma unroll
            for ( int u = 0; u < U; ++u ) l[u] = km_label_by_roots<KM>(xv[u], mu);
         }
         if ( i + U > all )
         {
#pragma unroll
            for ( int u = 0; u < U; ++u ) l[u] = i + u < lim ? l[u] : -1;
         }
#pragma unroll
         for ( int u = 0; u < U; ++u ) km_add<KM>(xv[u], l[u], s, n);
      }
   }
}

/*
 * computeLogLikelihood (pairwise_kmeans.cpp:106-127) of one run per lane, all of the pair in column c: one
 * accumulator, cluster by cluster in sample order.  The first sweep adds the samples of cluster 0 and leaves
 * labels and squared distances (ya, dbuf: this lane's interleaved columns) for the others'.  a: the means the
 * labels were assigned with, f: the final ones.
 */
template <int KT>
__device__ __forceinline__ float km_loglik(const float2* x, int N, int K, const F2 (&a)[KT], const F2 (&f)[KT], F2 z,
                                           int8_t* ya, float* dbuf)
{
   constexpr int U = 4;
   float S = 0.f;
#pragma unroll 1
   for ( int i = 0; i < N; i += U )
   {
      F2 xv[U];
      int l[U];
#pragma unroll
      for ( int u = 0; u < U; ++u )
         xv[u].v = *reinterpret_cast<const unsigned long long*>(x + min(i + u, N - 1) * KM_COLS);
      bool near = false;
#pragma unroll
      for ( int u = 0; u < U; ++u ) l[u] = km_label<KT>(xv[u], a, z, near);
      if ( near )
      {
#pragma unroll
         for ( int u = 0; u < U; ++u ) l[u] = km_label_by_roots<KT>(xv[u], a);
      }
#pragma unroll
      for ( int u = 0; u < U; ++u )
      {
         F2 m = f[0];
#pragma unroll
         for ( int k = 1; k < KT; ++k ) m.v = l[u] == k ? f[k].v : m.v;
         const float d = sqrtf(km_square(xv[u], m, z));
         const float dd = d * d;
         if ( i + u < N )
         {
            S += l[u] == 0 ? dd : 0.f;    /* S >= 0: adding +0 leaves it as it is */
            ya[(i + u) * TILE] = (int8_t)l[u];
            dbuf[(i + u) * TILE] = dd;
         }
      }
   }
   const int last = __reduce_max_sync(0xffffffffu, K);
#pragma unroll 1
   for ( int k = 1; k < last; ++k )
   {
#pragma unroll 1
      for ( int i = 0; i < N; i += 2 * U )
      {
         float d[2 * U];
         int l[2 * U];
#pragma unroll
         for ( int u = 0; u < 2 * U; ++u )
         {
            const int at = min(i + u, N - 1) * TILE;
            l[u] = i + u < N ? ya[at] : -1;
            d[u] = dbuf[at];
         }
#pragma unroll
         for ( int u = 0; u < 2 * U; ++u ) S += l[u] == k ? d[u] : 0.f;
      }
   }
   return -S;
}

/* the pair's rand() draws, in the reference's order, modulo N (the LCG restarts at every fit) */
__device__ __forceinline__ void km_draws(const DevParams& P, const DevData& D, uint64_t qpos, int N, int32_t* draws,
                                         int lane)
{
   const int total = km_draws_per_pair(P.min_k, P.max_k);
   if ( P.rand_mode == 0 )
   {
      /* 31 outputs at a time: out[i] = s[i] + s[i + 28], and s[i + 28] is out[i - 3] from i = 3 on, so the
       * outputs are running sums of every third word */
      uint32_t s = warp_rng_state(D, qpos * (uint64_t)P.draws_per_pair, lane);
      for ( int d = 0; d < total; d += RNG_WORDS )
      {
         const uint32_t far = __shfl_sync(0xffffffffu, s, lane < 3 ? lane + 28 : lane);
         uint32_t v = s + (lane < 3 ? far : 0u);
#pragma unroll
         for ( int o = 3; o < 32; o *= 2 )
         {
            const uint32_t up = __shfl_up_sync(0xffffffffu, v, o);
            if ( lane >= o ) v += up;
         }
         s = v;
         if ( lane < RNG_WORDS && d + lane < total ) draws[d + lane] = (int32_t)(v >> 1) % N;
      }
   }
   else
   {
      for ( int K = P.min_k, d = 0; K <= P.max_k; d += 10 * K, ++K )
      {
         for ( int i = lane; i < 10 * K; i += 32 )
         {
            uint64_t lcg = 1;
            for ( int j = 0; j <= i; ++j ) lcg = lcg * 1103515245ull + 12345ull;
            draws[d + i] = (int32_t)((uint32_t)(lcg / 65536ull) % 32768u) % N;
         }
      }
   }
   __syncwarp();
}

/* a column of X as the outlier and correlation passes read it */
struct KmColumn
{
   const float2* x;
   __device__ __forceinline__ float2 operator()(int i) const { return x[i * KM_COLS]; }
};

/*
 * One warp: its scratch slot holds X [S][KM_COLS], per column the sample labels (where no output row takes
 * them), the draws and the records of the runs; the log-likelihood sweep's labels and distances.
 */
template <int KT>
__global__ void __launch_bounds__(WARPS_PER_BLOCK * 32, KINC_MIN_BLOCKS)
k_kmeans_pairs(DevParams P, DevData D, DevScratch W, DevBlock B, int smem_sort)
{
   extern __shared__ __align__(16) float smem[];
   constexpr int RS = km_record_floats<KT>();
   const int lane = threadIdx.x & 31;
   const int warp = threadIdx.x >> 5;
   const int64_t slot = blockIdx.x * (int64_t)(blockDim.x >> 5) + warp;
   const size_t tile = (size_t)P.S * TILE, open_pairs = (size_t)P.S * KM_COLS;
   const int kmin = P.min_k, kmax = P.max_k;
   const int runs = 10 * (kmax - kmin + 1);               /* of one pair */
   const int sweeps = kmin == 1 ? runs - 10 : runs;       /* of them with more than one cluster */

   float2* X = W.X + slot * open_pairs;
   int8_t* labels = W.lbl + slot * open_pairs;
   float* dbuf = W.lpx + slot * tile + lane;
   int8_t* ya = W.ya + slot * tile + lane;
   int32_t* draws = W.kmd + (size_t)slot * P.km_dmax * KM_COLS;
   float* rec = W.kmr + (size_t)slot * P.km_tmax * RS;
   float* ring = smem + (size_t)warp * P.smem_floats;
   float* sort = smem_sort ? ring : W.sortbuf + slot * (size_t)P.sort_floats;
   const F2 z = f2(P.neg_zero);
   const F2 absent = f2(__int_as_float(0x7fc00000));
   KmStream stream;
   stream.X = X;
   stream.ring = (uint32_t)__cvta_generic_to_shared(ring);
   stream.S = P.S;
   stream.lane = lane;

   /* column c's pair is kept by lane c: pair, usable count, runs handed out, runs not yet ended (-1: empty) */
   int64_t cp = 0;
   int cN = 0, cnext = 0, cleft = -1;
   bool drained = false;                                   /* the queue is empty */
   unsigned long long units = 0, fits = 0;

   /* this lane's run */
   bool active = false;
   int t = 0, j = 0, K = 0, N = 0, it = 0;
   F2 mu[KT];
   int nprev[KT];
#pragma unroll
   for ( int k = 0; k < KT; ++k )
   {
      mu[k] = absent;
      nprev[k] = -1;
   }

   auto label_row = [&](int64_t p, int c) {
      return B.outLabels ? B.outLabels + (p - B.start) * (int64_t)P.S : labels + (size_t)c * P.S;
   };

   /* the pair in column c (its runs ended): choice, labels, outliers, correlations */
   auto close = [&](int c) {
      const int64_t p = __shfl_sync(0xffffffffu, cp, c);
      const int n = __shfl_sync(0xffffffffu, cN, c);
      int8_t* lbl = label_row(p, c);
      const float2* x = X + c;
      float* r0 = rec + (size_t)c * runs * RS;
      int bestK = 0;
      if ( n >= P.min_samples )
      {
         for ( int b = 0; b < runs; b += TILE )
         {
            const int run = min(b + lane, runs - 1);
            const int k_run = km_run_k(kmax, run);
            const float* r = r0 + (size_t)run * RS;
            F2 a[KT], f[KT];
#pragma unroll
            for ( int k = 0; k < KT; ++k )
            {
               a[k] = k < k_run ? f2(r[2 * k], r[2 * k + 1]) : absent;
               f[k] = k < k_run ? f2(r[2 * KT + 2 * k], r[2 * KT + 2 * k + 1]) : absent;
            }
            const float logL = km_loglik<KT>(x, n, k_run, a, f, z, ya, dbuf);
            if ( b + lane < runs ) r0[(size_t)run * RS + 4 * KT] = logL;
         }
         __syncwarp();
         float bestValue = INFINITY;
         int best = -1;
         for ( int k = kmin; k <= kmax; ++k )
         {
            float bestL = -INFINITY;
            int bi = -1;
            for ( int init = 0; init < 10; ++init )
            {
               const int run = (kmax - k) * 10 + init;
               const float l = r0[(size_t)run * RS + 4 * KT];
               if ( bestL < l )
               {
                  bestL = l;
                  bi = run;
               }
            }
            const float value = criterion_value<false>(P, D, k, bestL, n, 0.f);
            if ( value < bestValue )
            {
               bestValue = value;
               bestK = k;
               best = bi;
            }
         }
         /* that run's labels over the sample positions i < n with a label >= 0, in order */
         if ( bestK > 0 && best >= 0 )
         {
            const float* r = r0 + (size_t)best * RS;
            F2 a[KT];
#pragma unroll
            for ( int k = 0; k < KT; ++k ) a[k] = k < bestK ? f2(r[2 * k], r[2 * k + 1]) : absent;
            for ( int base = 0, q = 0; base < n; base += 32 )
            {
               const int i = base + lane;
               const bool in = i < n && lbl[i] >= 0;
               const unsigned bal = __ballot_sync(0xffffffffu, in);
               if ( in )
               {
                  F2 xv;
                  xv.v = *reinterpret_cast<const unsigned long long*>(x + (q + __popc(bal & lanemask_lt())) * KM_COLS);
                  bool near = false;
                  int l = km_label<KT>(xv, a, z, near);
                  if ( near ) l = km_label_by_roots<KT>(xv, a);
                  lbl[i] = (int8_t)l;
               }
               q += __popc(bal);
            }
            __syncwarp();
         }
      }
      pair_finish(P, D, B, KmColumn { x }, sort, lbl, p, n, bestK, lane);
      if ( lane == c ) cleft = -1;
   };

   /* the queue's next pair into empty column c */
   auto open = [&](int c) {
      unsigned long long q = 0;
      if ( lane == 0 ) q = atomicAdd(B.tiles, 1ull);
      q = __shfl_sync(0xffffffffu, q, 0);
      if ( (int64_t)q >= B.size )
      {
         drained = true;
         return;
      }
      const int64_t p = B.start + (B.order ? B.order[q] : (int64_t)q);
      int32_t x, y;
      pair_xy(p, x, y);
      int8_t* lbl = label_row(p, c);
      const int n = pair_fetch(P, D, x, y, lbl, lane, [&](int i, float v0, float v1) { X[i * KM_COLS + c] = make_float2(v0, v1); });
      if ( lane == 0 && n != B.N[p - B.lo] ) atomicCAS(B.status, ST_OK, ST_BAD_RANK);
      if ( P.pre_out )
      {
         pair_mark_outliers(KmColumn { X + c }, n, sort, 0, lbl, 0, -7, lane);
         pair_mark_outliers(KmColumn { X + c }, n, sort, 1, lbl, 0, -7, lane);
      }
      if ( lane == c )
      {
         cp = p;
         cN = n;
         cnext = 0;
         cleft = n >= P.min_samples ? sweeps : 0;
      }
      if ( n >= P.min_samples )
      {
         int32_t* dr = draws + (size_t)c * P.km_dmax;
         km_draws(P, D, B.qpos && P.rand_mode == 0 ? B.qpos[p - B.start] : 0, n, dr, lane);
         fits += lane == 0 ? (unsigned long long)(kmax - kmin + 1) : 0;
         if ( kmin == 1 )
         {
            /* one cluster: every sample is in it, as at the start, so the run ends with the mean it drew */
            units += lane == 0 ? 10ull * n : 0;
            if ( lane < 10 )
            {
               const float2 m = X[dr[lane] * KM_COLS + c];
               float* r = rec + ((size_t)c * runs + sweeps + lane) * RS;
               r[0] = r[2 * KT] = m.x;
               r[1] = r[2 * KT + 1] = m.y;
            }
         }
         __syncwarp();
      }
   };

   for ( ;; )
   {
      /* pairs whose runs have ended are closed; free lanes take the open pairs' next runs, then the queue's
       * next pair is opened */
      for ( ;; )
      {
         const unsigned done = __ballot_sync(0xffffffffu, cleft == 0);
         if ( done )
         {
            close(__ffs((int)done) - 1);
            continue;
         }
         const unsigned freem = __ballot_sync(0xffffffffu, !active);
         if ( !freem ) break;
         const unsigned ready = __ballot_sync(0xffffffffu, cleft > 0 && cnext < sweeps);
         if ( !ready )
         {
            const unsigned empty = __ballot_sync(0xffffffffu, lane < KM_COLS && cleft < 0);
            if ( drained || !empty ) break;
            open(__ffs((int)empty) - 1);
            continue;
         }
         const int c = __ffs((int)ready) - 1;
         const int from = __shfl_sync(0xffffffffu, cnext, c);
         const int n = __shfl_sync(0xffffffffu, cN, c);
         const int give = min(sweeps - from, __popc(freem));
         const int rank = __popc(freem & lanemask_lt());
         if ( lane == c ) cnext = from + give;
         if ( !active && rank < give )
         {
            t = from + rank;
            j = c;
            K = km_run_k(kmax, t);
            N = n;
            const int32_t* dr = draws + (size_t)c * P.km_dmax + km_draw_offset(kmin, K, t % 10);
#pragma unroll
            for ( int k = 0; k < KT; ++k )
            {
               mu[k] = absent;
               nprev[k] = -1;
               if ( k < K ) mu[k].v = *reinterpret_cast<const unsigned long long*>(X + dr[k] * KM_COLS + c);
            }
            it = 0;
            active = true;
         }
      }
      if ( !__any_sync(0xffffffffu, active) ) break;

      /* one Lloyd iteration of every active lane's run, samples in lockstep */
      const int most = __reduce_max_sync(0xffffffffu, active ? N : 0);
      const int all = __reduce_min_sync(0xffffffffu, active ? N : 0x7fffffff);
      const int widest = __reduce_max_sync(0xffffffffu, active ? K : 0);
      F2 s[KT];
      int n[KT];
      auto sweep = [&](auto count) {
         constexpr int KM = decltype(count)::value;
         F2 m[KM], sums[KM];
         int cnt[KM];
#pragma unroll
         for ( int k = 0; k < KM; ++k ) m[k] = mu[k];
         km_sweep<KM>(stream, j, active ? N : 0, all, most, m, z, sums, cnt);
#pragma unroll
         for ( int k = 0; k < KT; ++k )
         {
            s[k] = k < KM ? sums[k < KM ? k : 0] : f2(0.f);
            n[k] = k < KM ? cnt[k < KM ? k : 0] : 0;
         }
      };
      if ( widest <= 2 )
         sweep(std::integral_constant<int, 2>());
      else if ( KT == 3 || widest == 3 )
         sweep(std::integral_constant<int, 3>());
      else
         sweep(std::integral_constant<int, KT>());
      bool ended = false;
      if ( active )
      {
         units += (unsigned long long)N * K;
         /*
          * "no label changed", without the labels.  First iteration: they were all zero, so unchanged <=>
          * every sample in cluster 0.  Later: unchanged labels give the same sums and so the same means and
          * counts; and if means and counts are the same although labels changed, the next iteration assigns
          * by the same means, changes nothing and ends with what this one has.
          */
         F2 nm[KT];
         bool same = true;
#pragma unroll
         for ( int k = 0; k < KT; ++k )
         {
            nm[k] = absent;
            if ( k >= K ) continue;
            const float sc = 1.0f / n[k];
            nm[k] = f2(lo(s[k]) * sc, hi(s[k]) * sc);
            same = same && nm[k].v == mu[k].v && n[k] == nprev[k];
         }
         if ( it == 0 ) same = n[0] == N;
         ended = same || it == 299;
         if ( ended )
         {
            /* converged: the labels were assigned with the current means, which stay; out of iterations:
             * the means then moved once more */
            float* r = rec + ((size_t)j * runs + t) * RS;
#pragma unroll
            for ( int k = 0; k < KT; ++k )
            {
               if ( k >= K ) continue;
               const F2 last = same ? mu[k] : nm[k];
               r[2 * k] = lo(mu[k]); r[2 * k + 1] = hi(mu[k]);
               r[2 * KT + 2 * k] = lo(last); r[2 * KT + 2 * k + 1] = hi(last);
            }
            active = false;
         }
         ++it;
#pragma unroll
         for ( int k = 0; k < KT; ++k )
         {
            mu[k] = nm[k];
            nprev[k] = n[k];
         }
      }
      /* the columns of the runs that ended */
      for ( unsigned m = __ballot_sync(0xffffffffu, ended); m; m &= m - 1u )
      {
         const int c = __shfl_sync(0xffffffffu, j, __ffs((int)m) - 1);
         if ( lane == c ) --cleft;
      }
      __syncwarp();
   }
   for ( int o = 16; o > 0; o >>= 1 )
   {
      units += __shfl_xor_sync(0xffffffffu, units, o);
      fits += __shfl_xor_sync(0xffffffffu, fits, o);
   }
   if ( lane == 0 && B.work )
   {
      atomicAdd(&B.work[0], units);
      atomicAdd(&B.work[1], fits);
   }
}

} /* namespace kinc */
