/* Similarity without clustering (clusmethod none): Pearson from the rows of the matrix, Spearman from every
 * gene's sample order, and the tile kernel's specialisation for what is left. */
#include "sim_pair.cuh"

#include <algorithm>
#include <cmath>

namespace kinc {

SimKernel sim_kernel_none()
{
   return sim_kernel_handle<0, 0>();
}

cudaError_t sim_launch_none(const SimKernel&, int grid, int smem, cudaStream_t st, const DevParams& P,
                            const DevData& D, const DevScratch& W, const DevBlock& B, int smem_sort)
{
   return sim_kernel_launch<0, 0>(grid, smem, st, P, D, W, B, smem_sort);
}

/*
 * Pearson without clustering (K = 1), one thread per pair, straight from the expression rows and
 * the usable-sample masks -- no compaction into scratch, no labels (rows with K <= 1 carry none).
 * Without clustering a sample position's label is 0 exactly when both genes' values are usable,
 * so Pearson::computeCluster (pairwise_pearson.cpp:12-52) reduces to: for every usable position i,
 * in order, add the point the reference reads there -- semantics 0: its packed array at i, which
 * for i < N is the pair's own i-th usable sample and for i >= N what the last earlier pair of the
 * work block with more than i usable samples left (the k_links links; zero if none); semantics 1:
 * sample i itself.  Same sums in the same order as lane_pearson, so the same bits.
 */
__global__ void __launch_bounds__(256) k_pearson_lanes(DevParams P, DevData D, DevBlock B)
{
   const int64_t stride = (int64_t)gridDim.x * blockDim.x;
   for ( int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < B.size; q += stride )
   {
      const int64_t p = B.start + q;
      int32_t x, y;
      pair_xy(p, x, y);
      const uint32_t* mx = D.umask + (size_t)x * P.W;
      const uint32_t* my = D.umask + (size_t)y * P.W;
      const float* g1 = D.gem + (size_t)x * P.S;
      const float* g2 = D.gem + (size_t)y * P.S;
      int n = 0;
      float sumx = 0, sumy = 0, sumx2 = 0, sumy2 = 0, sumxy = 0;
      auto add = [&](float vx, float vy) {
         sumx += vx; sumy += vy; sumx2 += vx * vx; sumy2 += vy * vy; sumxy += vx * vy;
         ++n;
      };
      if ( P.semantics == 0 )
      {
         const int N = B.N[p - B.lo];
         /* positions i < N: i-th usable sample (cursor s) where position i is usable */
         int ws = 0;
         uint32_t bs = __ldg(mx) & __ldg(my);
         for ( int w = 0; w * 32 < N; ++w )
         {
            const uint32_t pos = __ldg(mx + w) & __ldg(my + w);
            const int hi = min(32, N - w * 32);
            for ( int b = 0; b < hi; ++b )
            {
               while ( bs == 0 && ws + 1 < P.W )
               {
                  ++ws;
                  bs = __ldg(mx + ws) & __ldg(my + ws);
               }
               const int s = ws * 32 + __ffs(bs) - 1;
               bs &= bs - 1;
               /* an unusable position adds +0.0, which leaves every sum as it is (a sum of floats
                * starting at +0.0 is never -0.0), so the lanes need not branch */
               const bool use = (pos >> b) & 1u;
               const float vx = use ? __ldg(g1 + s) : 0.f;
               const float vy = use ? __ldg(g2 + s) : 0.f;
               sumx += vx; sumy += vy; sumx2 += vx * vx; sumy2 += vy * vy; sumxy += vx * vy;
               n += use;
            }
         }
         /* positions i >= N: stale points of earlier pairs of the work block (as lane_pearson) */
         const int32_t self = (int32_t)(p - B.lo);
         int32_t c = B.pg[self];
         if ( c >= self ) c = -1;
         PackedCursor cur;
         for ( int w = N >> 5; w < P.W; ++w )
         {
            uint32_t pos = __ldg(mx + w) & __ldg(my + w);
            if ( w == (N >> 5) ) pos &= ~0u << (N & 31);
            while ( pos )
            {
               const int i = w * 32 + __ffs(pos) - 1;
               pos &= pos - 1;
               while ( c >= 0 && B.N[c] <= i )
               {
                  const int32_t nxt = B.pg[c];
                  c = nxt < c ? nxt : -1;
               }
               const float2 v = c >= 0 ? cur.at(P, D, B.lo + c, i) : make_float2(0.f, 0.f);
               add(v.x, v.y);
            }
         }
      }
      else
      {
         for ( int w = 0; w < P.W; ++w )
         {
            uint32_t pos = __ldg(mx + w) & __ldg(my + w);
            while ( pos )
            {
               const int i = w * 32 + __ffs(pos) - 1;
               pos &= pos - 1;
               add(__ldg(g1 + i), __ldg(g2 + i));
            }
         }
      }
      const float r = pearson_value(P, n, sumx, sumy, sumx2, sumy2, sumxy);
      if ( B.outK ) B.outK[q] = 1;
      if ( B.outCorr )
      {
         float* row = B.outCorr + q * P.max_k * P.ncorr;
         row[0] = r;
         for ( int k = 1; k < P.max_k * P.ncorr; ++k ) row[k] = __int_as_float(0x7fc00000);
      }
   }
}

static cudaError_t sim_launch_pearson_lanes(int sms, cudaStream_t st, const DevParams& P, const DevData& D,
                                     const DevBlock& B)
{
   const int64_t blocks = std::min<int64_t>((B.size + 255) / 256, (int64_t)sms * 16);
   k_pearson_lanes<<<(int)std::max<int64_t>(1, blocks), 256, 0, st>>>(P, D, B);
   return cudaGetLastError();
}

/*
 * The same on tiles of genes: the threads of a CTA share the tile's values in shared memory, 32 samples at a time and
 * zero where unusable, and each sums R x R pairs (R genes x, R genes y) in registers.  Which samples a pair adds is a
 * bit mask per 32 samples: the usable ones, or with semantics 0 those of them whose rank is itself a usable position
 * (the r-th usable sample is read at position r), so every addition is one predicated instruction.  The points that
 * positions i >= N read follow: the chain of earlier pairs with larger counts N_c, each giving its last N_c - i usable
 * samples.
 *
 * One thread per pair straight from the matrix rows (k_pearson_lanes) issues 49 instructions per sample and touches
 * 32 rows per load.  R = 2 issues 9 to 11 (5 predicated additions, the bit test, the products) and keeps 0.85 of the
 * issue slots busy; R = 1 issues more but has four times the threads, which blocks of few pairs, and the walks along
 * the chain, need.  The choice and its times: sim_launch_pearson.
 */
constexpr int PT_THREADS = 128;
constexpr int PT_SMEM = 100 * 1024;         /* dynamic shared memory at most; the kernels' limit, the same for every caller
                                               (it belongs to the kernel, not to a context) */

/* a tile of TX genes x and as many y as make R x R pairs a thread; few rows x take flat tiles */
template <int TX, int R>
struct PearsonTile
{
   static constexpr int X = TX, Y = R * R * PT_THREADS / TX;
   static constexpr int GENES = X + Y;
   static constexpr int ROW = GENES + 2;    /* floats between samples */
   static size_t bytes(int W) { return (size_t)(32 * ROW + GENES * W) * sizeof(float); }
};

/* bits moved, in order, to the set positions of u */
__device__ __forceinline__ uint32_t deposit_bits(uint32_t bits, uint32_t u)
{
   /* make room at every clear position, from the lowest up */
   uint32_t clear = ~u;
   while ( clear )
   {
      const uint32_t below = (clear & (0u - clear)) - 1u;
      bits = (bits & below) | ((bits & ~below) << 1);
      clear &= clear - 1u;
   }
   return bits;
}

/* the five sums of a pair */
struct PearsonSums
{
   float x = 0.f, y = 0.f, xx = 0.f, yy = 0.f, xy = 0.f;
};

/* a thread's values of a sample and their squares */
template <int R>
__device__ __forceinline__ void pearson_values(const float* v, float (&x)[R], float (&xx)[R])
{
   if constexpr ( R == 2 )
   {
      const float2 q = *reinterpret_cast<const float2*>(v);
      x[0] = q.x;
      x[1] = q.y;
   }
   else
      x[0] = *v;
#pragma unroll
   for ( int a = 0; a < R; ++a ) xx[a] = x[a] * x[a];
}

/* one sample added if bit `b` of `in` is set */
__device__ __forceinline__ void pearson_add(PearsonSums& s, uint32_t in, int b, float vx, float vy, float vxx, float vyy,
                                            float vxy)
{
   asm("{\n\t.reg .pred p;\n\t.reg .b32 t;\n\tand.b32 t, %5, %6;\n\tsetp.ne.u32 p, t, 0;\n\t"
       "@p add.rn.f32 %0, %0, %7;\n\t@p add.rn.f32 %1, %1, %8;\n\t@p add.rn.f32 %2, %2, %9;\n\t"
       "@p add.rn.f32 %3, %3, %10;\n\t@p add.rn.f32 %4, %4, %11;\n\t}"
       : "+f"(s.x), "+f"(s.y), "+f"(s.xx), "+f"(s.yy), "+f"(s.xy)
       : "r"(in), "r"(1u << b), "f"(vx), "f"(vy), "f"(vxx), "f"(vyy), "f"(vxy));
}

/* positions i >= N: what the last earlier pair of the work block with more than i usable samples left there.
 * Pair p = (x, y) of B.lo's span; mx, my: its genes' masks.  (Slower, for all pairs of 1,000 x 200: one flat loop
 * over the pair's positions, so that the lanes of a warp advance together, 186 us against 166; four points in
 * flight, 176 us.) */
__device__ inline void pearson_stale(const DevParams& P, const DevData& D, const DevBlock& B, int64_t p, int32_t x, int N,
                                     const uint32_t* mx, const uint32_t* my, PearsonSums& sums)
{
   const int32_t self = (int32_t)(p - B.lo);
   const int64_t row0 = (int64_t)x * (x - 1) / 2;
   int32_t c = B.pg[self];
   /* links point strictly backwards; anything else ends the walk */
   if ( c >= self ) c = -1;
   int i = N;
   while ( c >= 0 )
   {
      const int Nc = B.N[c];
      const int32_t next = B.pg[c];
      const int64_t pc = B.lo + c;
      int32_t xc = x, yc = (int32_t)(pc - row0);
      if ( pc < row0 ) pair_xy(pc, xc, yc);
      const uint32_t* ux = D.umask + (size_t)xc * P.W;
      const uint32_t* uy = D.umask + (size_t)yc * P.W;
      const float* g1 = D.gem + (size_t)xc * P.S;
      const float* g2 = D.gem + (size_t)yc * P.S;
      /* its samples of rank i..Nc-1 are its last Nc - i: found from the end */
      int w = P.W - 1, left = Nc - i;
      uint32_t m = __ldg(ux + w) & __ldg(uy + w);
      while ( __popc(m) < left && w > 0 )
      {
         left -= __popc(m);
         --w;
         m = __ldg(ux + w) & __ldg(uy + w);
      }
      uint32_t low = m;
      for ( ; left > 0 && low; --left ) low &= ~(0x80000000u >> __clz((int)low));
      m &= ~low;
      for ( ; i < Nc; ++i )
      {
         while ( !m && w + 1 < P.W )
         {
            ++w;
            m = __ldg(ux + w) & __ldg(uy + w);
         }
         const int s = w * 32 + __ffs((int)m) - 1;
         m &= m - 1u;
         if ( ((mx[i >> 5] & my[i >> 5]) >> (i & 31)) & 1u )
         {
            const float vx = __ldg(g1 + s), vy = __ldg(g2 + s);
            sums.x += vx;
            sums.y += vy;
            sums.xx += vx * vx;
            sums.yy += vy * vy;
            sums.xy += vx * vy;
         }
      }
      c = next < c ? next : -1;
   }
   /* beyond the longest of them the array still holds zeros, which change no sum */
}

template <int TX, int R>
__global__ void __launch_bounds__(PT_THREADS)
k_pearson_tiles(DevParams P, DevData D, DevBlock B, int x0)
{
   using T = PearsonTile<TX, R>;
   constexpr int PT_X = T::X, PT_Y = T::Y, PT_GENES = T::GENES, PT_ROW = T::ROW;
   extern __shared__ __align__(16) float pt_smem[];
   float* v = pt_smem;                                            /* [32][PT_ROW] */
   uint32_t* mask = (uint32_t*)(pt_smem + 32 * PT_ROW);           /* [PT_GENES][W] */
   const int gx = x0 + blockIdx.y * PT_X, gy = blockIdx.x * PT_Y;
   /* pairs (x, y), x > y, of [start, end): nothing here? */
   const int xl = min(gx + PT_X - 1, P.G - 1);
   if ( gy >= xl ) return;
   {
      const int64_t first = (int64_t)gx * (gx - 1) / 2 + gy, last = (int64_t)xl * (xl - 1) / 2 + min(gy + PT_Y - 1, xl - 1);
      if ( last < B.start || first >= B.start + B.size ) return;
   }
   const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
   const int tx = R * (tid / (PT_Y / R)), ty = R * (tid % (PT_Y / R));
   auto gene = [&](int i) { return i < PT_X ? gx + i : gy + i - PT_X; };
   for ( int i = tid; i < PT_GENES * P.W; i += PT_THREADS )
   {
      const int g = gene(i / P.W);
      mask[i] = g < P.G ? __ldg(D.umask + (size_t)g * P.W + i % P.W) : 0u;
   }
   /* the next 32 samples of the tile on their way in registers: gene warp + 4k, sample lane */
   constexpr int PER = (PT_GENES + PT_THREADS / 32 - 1) / (PT_THREADS / 32);
   float next[PER];
   auto fetch = [&](int w) {
      const int s = w * 32 + lane;
#pragma unroll
      for ( int k = 0; k < PER; ++k )
      {
         const int i = warp + k * (PT_THREADS / 32), g = gene(i);
         next[k] = i < PT_GENES && g < P.G && s < P.S ? __ldg(D.gem + (size_t)g * P.S + s) : 0.f;
      }
   };
   fetch(0);
   __syncthreads();

   const uint32_t *mx[R], *my[R];
   PearsonSums sums[R][R];
   int n[R][R];
#pragma unroll
   for ( int a = 0; a < R; ++a )
   {
      mx[a] = mask + (tx + a) * P.W;
      my[a] = mask + (PT_X + ty + a) * P.W;
#pragma unroll
      for ( int b = 0; b < R; ++b ) n[a][b] = 0;
   }
   for ( int w = 0; w < P.W; ++w )
   {
#pragma unroll
      for ( int k = 0; k < PER; ++k )
      {
         const int i = warp + k * (PT_THREADS / 32);
         if ( i < PT_GENES ) v[lane * PT_ROW + i] = (mask[i * P.W + w] >> lane) & 1u ? next[k] : 0.f;
      }
      __syncthreads();
      if ( w + 1 < P.W ) fetch(w + 1);
      uint32_t in[R][R];
#pragma unroll
      for ( int a = 0; a < R; ++a )
#pragma unroll
         for ( int b = 0; b < R; ++b )
         {
            const uint32_t u = mx[a][w] & my[b][w];
            uint32_t take = u;
            if ( P.semantics == 0 )
            {
               const int r = n[a][b], k = r >> 5, k1 = min(k + 1, P.W - 1);
               take = deposit_bits(__funnelshift_r(mx[a][k] & my[b][k], mx[a][k1] & my[b][k1], r & 31), u);
            }
            in[a][b] = take;
            n[a][b] += __popc(u);
         }
#pragma unroll 8
      for ( int s = 0; s < 32; ++s )
      {
         float xs[R], ys[R], xq[R], yq[R];
         pearson_values(v + s * PT_ROW + tx, xs, xq);
         pearson_values(v + s * PT_ROW + PT_X + ty, ys, yq);
#pragma unroll
         for ( int a = 0; a < R; ++a )
#pragma unroll
            for ( int b = 0; b < R; ++b ) pearson_add(sums[a][b], in[a][b], s, xs[a], ys[b], xq[a], yq[b], xs[a] * ys[b]);
      }
      __syncthreads();
   }
#pragma unroll
   for ( int a = 0; a < R; ++a )
#pragma unroll
      for ( int b = 0; b < R; ++b )
      {
         const int x = gx + tx + a, y = gy + ty + b;
         if ( x >= P.G || y >= x ) continue;
         const int64_t p = (int64_t)x * (x - 1) / 2 + y, q = p - B.start;
         if ( q < 0 || q >= B.size ) continue;
         PearsonSums t = sums[a][b];
         if ( P.semantics == 0 && n[a][b] < P.S ) pearson_stale(P, D, B, p, x, n[a][b], mx[a], my[b], t);
         const float r = pearson_value(P, n[a][b], t.x, t.y, t.xx, t.yy, t.xy);
         if ( B.outK ) B.outK[q] = 1;
         if ( B.outCorr )
         {
            float* row = B.outCorr + q * P.max_k * P.ncorr;
            row[0] = r;
            for ( int k = 1; k < P.max_k * P.ncorr; ++k ) row[k] = __int_as_float(0x7fc00000);
         }
      }
}

template <int TX, int R>
static cudaError_t launch_pearson_tiles(cudaStream_t st, const DevParams& P, const DevData& D, const DevBlock& B, int x0,
                                        int x1)
{
   using T = PearsonTile<TX, R>;
   const int smem = (int)T::bytes(P.W);
   /* 48 KB need no leave (the call costs a microsecond) */
   const cudaError_t e = smem <= 48 * 1024 ? cudaSuccess
      : cudaFuncSetAttribute(k_pearson_tiles<TX, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, PT_SMEM);
   if ( e != cudaSuccess ) return e;
   const dim3 grid((x1 + T::Y - 1) / T::Y, (x1 - x0) / TX + 1);
   k_pearson_tiles<TX, R><<<grid, PT_THREADS, smem, st>>>(P, D, B, x0);
   return cudaGetLastError();
}

/* whether the masks of a tile's genes fit in shared memory beside 32 samples of their values */
template <int TX, int R>
static bool pearson_tiles_fit(const DevParams& P)
{
   return PearsonTile<TX, R>::bytes(P.W) <= (size_t)PT_SMEM;
}

/*
 * Microseconds, k_pearson_lanes / R = 1 / R = 2 (with the launches before them), by the mean N of a pair over S:
 *   1,000 samples, own values      1 pair, 0.9: 81 / 51 / 122      500 pairs: 143 / 53 / 125     32,768: 154 / 44 / 73
 *                                  131,072: 259 / 112 / 102        499,500: 899 / 326 / 260
 *   1,000 samples, packed reads    1 pair, 0.9: 121 / 60 / 154     500 pairs: 393 / 80 / 193     32,768: 514 / 90 / 201
 *                                  499,500, 0.9: 1,967 / 518 / 527    1,048,576: 3,837 / 1,001 / 940
 *                                  32,768, 0.49: 1,713 / 683 / 2,093  1,048,576: 9,499 / 3,915 / 5,004
 *   lanes pass over what a pair lacks, tiles do not: own values, 262,144 pairs, 0.25: 234 / 179 / 184; 0.04: 123 / 179 /
 *   180; packed reads 0.25: 727 / 376 / 495, 0.04: 215 / 341 / 452; one pair, packed reads 0.49: 96 / 70 / 193, 0.25:
 *   56 / 72 / 199.
 * So lanes where a pair has less than an eighth of the samples (a few pairs: a third), R = 2 from 120,000 pairs with own
 * values and from 900,000 with packed reads and little missing, R = 1 elsewhere.
 */
cudaError_t sim_launch_pearson(int sms, cudaStream_t st, const DevParams& P, const DevData& D, const DevBlock& B, double n)
{
   /* the rows x of the block */
   auto row_of = [](int64_t p) {
      int64_t x = (int64_t)((1.0 + std::sqrt(1.0 + 8.0 * (double)p)) / 2.0);
      while ( x * (x - 1) / 2 > p ) --x;
      while ( (x + 1) * x / 2 <= p ) ++x;
      return (int)x;
   };
   const int x0 = row_of(B.start), x1 = row_of(B.start + B.size - 1), rows = x1 - x0 + 1;
   const double share = n / P.S;
   if ( share < (B.size < 8 ? 0.35 : 0.125) ) return sim_launch_pearson_lanes(sms, st, P, D, B);
   const bool many = P.semantics != 0 ? B.size >= 120000 : B.size >= 900000 && share >= 0.75;
   if ( many && rows > 8 && pearson_tiles_fit<16, 2>(P) ) return launch_pearson_tiles<16, 2>(st, P, D, B, x0, x1);
   if ( many && rows > 2 && pearson_tiles_fit<4, 2>(P) ) return launch_pearson_tiles<4, 2>(st, P, D, B, x0, x1);
   /* tiles of 2 x 64, 4 x 32 or 8 x 16 genes */
   if ( rows <= 2 && pearson_tiles_fit<2, 1>(P) ) return launch_pearson_tiles<2, 1>(st, P, D, B, x0, x1);
   if ( rows <= 6 && pearson_tiles_fit<4, 1>(P) ) return launch_pearson_tiles<4, 1>(st, P, D, B, x0, x1);
   if ( pearson_tiles_fit<8, 1>(P) ) return launch_pearson_tiles<8, 1>(st, P, D, B, x0, x1);
   return sim_launch_pearson_lanes(sms, st, P, D, B);
}

/*
 * Spearman without clustering.  Spearman::computeCluster (pairwise_spearman.cpp:27-86) sorts the pair's
 * usable samples by x, then by y, and sums the squared differences of the two ranks.  The ranks among the
 * samples that both genes have follow from each gene's own sample order: walked in that order, a sample's
 * rank is the number of samples before it that the other gene has too.  So every gene is sorted once per
 * matrix (k_gene_order), and a pair costs two walks of S / 32 warp steps instead of two sorting networks:
 * 262,144 pairs of 1,000 samples (10 % missing) 32.8 -> 1.7 ms, half of it the pairs of the next paragraph.
 *
 * Where two equal values of a gene both take part, their order comes from the network's swaps; the walk
 * finds such pairs (a flag per sample: equal to the next in order) and lists them for a launch of their own,
 * a network per CTA of one warp in shared memory.  (In the walking warps they took 4 ms of 5: a gene with a
 * repeated value gives a run of them to one warp.)
 */
constexpr int ORDER_THREADS = 256;
constexpr int ORDER_MOST = 8192;            /* samples k_gene_order sorts in shared memory (64 KB of keys) */
constexpr uint16_t ORDER_TIE = 0x8000;
constexpr int SPEARMAN_WARPS = 8;
/* dynamic shared memory at ORDER_MOST samples: the kernels' limits, the same for every caller (they belong to the
 * kernels, not to a context) */
constexpr int ORDER_SMEM = ORDER_MOST * (int)sizeof(unsigned long long);
constexpr int SPEARMAN_SMEM = SPEARMAN_WARPS * (ORDER_MOST / 8 + ORDER_MOST * (int)sizeof(uint16_t));
constexpr int TIES_SMEM = ORDER_MOST / 8 + 2 * ORDER_MOST * (int)sizeof(float);

/* order[g][r]: the r-th of gene g's usable samples by value, ORDER_TIE set if the next one is equal; filled up
 * with samples the gene lacks.  ties[g]: 1 if any is set, 2 added if the gene has +inf, with which the network
 * fills its buffers up. */
__global__ void __launch_bounds__(ORDER_THREADS)
k_gene_order(const float* __restrict__ gem, const uint32_t* __restrict__ umask, int G, int S, int W, int P2,
             uint16_t* __restrict__ order, uint8_t* __restrict__ ties)
{
   extern __shared__ unsigned long long key[];
   for ( int g = blockIdx.x; g < G; g += gridDim.x )
   {
      for ( int i = threadIdx.x; i < P2; i += ORDER_THREADS )
      {
         unsigned long long k = ~0ull << 16;
         if ( i < S && ((umask[(size_t)g * W + (i >> 5)] >> (i & 31)) & 1u) )
         {
            const float v = gem[(size_t)g * S + i];
            const uint32_t b = v == 0.f ? 0u : __float_as_uint(v);
            k = (unsigned long long)(b & 0x80000000u ? ~b : b | 0x80000000u) << 16;
         }
         key[i] = k | (unsigned)i;
      }
      __syncthreads();
      for ( int ob = 2; ob <= P2; ob *= 2 )
      {
         for ( int t = ob / 2; t >= 1; t /= 2 )
         {
            for ( int i = threadIdx.x; i < P2 / 2; i += ORDER_THREADS )
            {
               const int a = (i / t) * 2 * t + i % t, b = a + t;
               const bool up = !(a & ob);
               const unsigned long long ka = key[a], kb = key[b];
               if ( (ka > kb) == up )
               {
                  key[a] = kb;
                  key[b] = ka;
               }
            }
            __syncthreads();
         }
      }
      int any = 0;
      for ( int i = threadIdx.x; i < S; i += ORDER_THREADS )
      {
         const unsigned long long k = key[i] >> 16;
         const bool usable = k <= 0xffffffffull;
         const bool tie = usable && i + 1 < S && key[i + 1] >> 16 == k;
         order[(size_t)g * S + i] = (uint16_t)((key[i] & 0x7fffu) | (tie ? ORDER_TIE : 0));
         any |= (tie ? 1 : 0) | (k == 0xff800000ull ? 2 : 0);
      }
      const int tied = __syncthreads_or(any & 1), inf = __syncthreads_or(any & 2);
      if ( threadIdx.x == 0 ) ties[g] = (uint8_t)((tied ? 1 : 0) | (inf ? 2 : 0));
   }
}

bool sim_spearman_orders_fit(const DevParams& P)
{
   return P.clus == 0 && P.corr >= 1 && P.S <= ORDER_MOST;
}

size_t sim_spearman_orders_bytes(const DevParams& P, char* base, SpearmanOrders* out)
{
   const size_t order = ((size_t)P.G * P.S * sizeof(uint16_t) + 255) & ~(size_t)255;
   if ( out ) *out = SpearmanOrders { (uint16_t*)base, (uint8_t*)(base + order), 0, 0, 0, 0 };
   return order + (size_t)P.G;
}

/*
 * One walk: the samples of `order` that `mask` (shared memory) has, in order; use(sample, rank).  With `check`,
 * *tied is set when two of them are equal in value.
 */
template <bool CHECK, class Use>
__device__ __forceinline__ int spearman_walk(const uint16_t* __restrict__ order, int S, const uint32_t* mask, int lane,
                                             bool& tied, Use use)
{
   constexpr int U = 4;
   int n = 0;
   bool open = false;                       /* the last sample taken is equal to all that followed it so far */
   for ( int base = 0; base < S; base += 32 * U )
   {
      uint32_t o[U];
#pragma unroll
      for ( int u = 0; u < U; ++u )
      {
         const int i = base + u * 32 + lane;
         o[u] = i < S ? __ldg(order + i) : 0xffffffffu;
      }
#pragma unroll
      for ( int u = 0; u < U; ++u )
      {
         const uint32_t s = o[u] & 0x7fffu;
         const bool in = o[u] != 0xffffffffu && ((mask[s >> 5] >> (s & 31)) & 1u);
         const unsigned bal = __ballot_sync(0xffffffffu, in);
         if ( in ) use((int)s, n + __popc(bal & lanemask_lt()));
         n += __popc(bal);
         if ( CHECK )
         {
            const unsigned eq = __ballot_sync(0xffffffffu, o[u] != 0xffffffffu && (o[u] & ORDER_TIE));
            /* the samples equal to this lane's run up to the first that is not flagged */
            const unsigned rest = ~(eq >> lane);
            const int len = rest ? __ffs((int)rest) - 1 : 32;      /* flagged in a row from this lane on */
            const unsigned reach = len >= 31 ? 0xfffffffeu : (2u << len) - 2u;
            bool t = in && ((bal >> lane) & reach);
            if ( lane == 0 && open && bal )
            {
               const int first = __ffs((int)bal) - 1;
               t = t || (eq & ((1u << first) - 1u)) == (1u << first) - 1u;
            }
            tied = tied || __any_sync(0xffffffffu, t);
            if ( bal )
            {
               const int last = 31 - __clz((int)bal);
               open = (eq >> last) == (0xffffffffu >> last);
            }
            else
            {
               open = open && eq == 0xffffffffu;
            }
         }
      }
   }
   return n;
}

__global__ void __launch_bounds__(SPEARMAN_WARPS * 32)
k_spearman_orders(DevParams P, DevData D, DevBlock B, SpearmanOrders R, int32_t* tied_pairs, int warp_bytes, int per_warp)
{
   extern __shared__ __align__(16) unsigned char spearman_smem[];
   const int lane = threadIdx.x & 31;
   const int warp = threadIdx.x >> 5;
   unsigned char* base = spearman_smem + (size_t)warp * warp_bytes;
   uint32_t* mask = (uint32_t*)base;                                     /* samples that both genes have */
   uint16_t* ranks = (uint16_t*)(base + ((P.W * 4 + 15) & ~15));         /* by x */
   const int c = P.corr == 2 ? 1 : 0;
   const float nan = __int_as_float(0x7fc00000);
   const int64_t step = (int64_t)gridDim.x * SPEARMAN_WARPS * per_warp;
   for ( int64_t q0 = ((int64_t)blockIdx.x * SPEARMAN_WARPS + warp) * per_warp; q0 < B.size; q0 += step )
   {
      int32_t x, y;
      pair_xy(B.start + q0, x, y);
      for ( int64_t q = q0; q < min(q0 + per_warp, B.size); ++q )
      {
         if ( B.outLabels )
         {
            const float* g1 = D.gem + (size_t)x * P.S;
            const float* g2 = D.gem + (size_t)y * P.S;
            int8_t* row = B.outLabels + q * (int64_t)P.S;
            for ( int i = lane; i < P.S; i += 32 )
            {
               const float v1 = __ldg(g1 + i), v2 = __ldg(g2 + i);
               row[i] = isnan(v1) || isnan(v2) ? (int8_t)-9 : v1 < P.min_expr || v2 < P.min_expr ? (int8_t)-6 : (int8_t)0;
            }
         }
         const uint32_t* mx = D.umask + (size_t)x * P.W;
         const uint32_t* my = D.umask + (size_t)y * P.W;
         for ( int w = lane; w < P.W; w += 32 ) mask[w] = __ldg(mx + w) & __ldg(my + w);
         __syncwarp();
         float r = nan;
         const int tx = R.ties[x], ty = R.ties[y];
         bool tied = ((tx | ty) & 2) != 0;
         int n;
         auto rank = [&](int s, int i) { ranks[s] = (uint16_t)i; };
         if ( tx )
            n = spearman_walk<true>(R.order + (size_t)x * P.S, P.S, mask, lane, tied, rank);
         else
            n = spearman_walk<false>(R.order + (size_t)x * P.S, P.S, mask, lane, tied, rank);
         __syncwarp();
         if ( n >= P.min_samples )
         {
            uint32_t diff = 0;
            auto add = [&](int s, int i) {
               const int d = i - (int)ranks[s];
               diff += (uint32_t)(d * d);
            };
            if ( ty )
               spearman_walk<true>(R.order + (size_t)y * P.S, P.S, mask, lane, tied, add);
            else
               spearman_walk<false>(R.order + (size_t)y * P.S, P.S, mask, lane, tied, add);
            r = spearman_value(__reduce_add_sync(0xffffffffu, diff), n);
            if ( tied && lane == 0 ) tied_pairs[atomicAdd(B.tiles, 1ull)] = (int32_t)q;
         }
         __syncwarp();
         float* row = B.outCorr ? B.outCorr + q * P.max_k * P.ncorr : nullptr;
         if ( row )
         {
            if ( P.ncorr == 1 )
            {
               for ( int k = lane; k < P.max_k; k += 32 ) row[k] = k == 0 ? r : nan;
            }
            else if ( lane == 0 )
            {
               row[c] = r;                  /* the Pearson kernel has filled the rest */
            }
         }
         if ( lane == 0 && B.outK ) B.outK[q] = 1;
         if ( ++y >= x )
         {
            y = 0;
            ++x;
         }
      }
   }
}

/* the pairs whose ranks the network decides, one per warp (and CTA) */
__global__ void __launch_bounds__(32) k_spearman_ties(DevParams P, DevData D, DevBlock B, const int32_t* tied_pairs)
{
   extern __shared__ __align__(16) unsigned char spearman_smem[];
   const int lane = threadIdx.x;
   uint32_t* mask = (uint32_t*)spearman_smem;
   float* buf = (float*)(spearman_smem + ((P.W * 4 + 15) & ~15));
   const int64_t count = (int64_t)*B.tiles;
   for ( int64_t i = blockIdx.x; i < count; i += gridDim.x )
   {
      const int64_t q = tied_pairs[i];
      int32_t x, y;
      pair_xy(B.start + q, x, y);
      for ( int w = lane; w < P.W; w += 32 ) mask[w] = __ldg(D.umask + (size_t)x * P.W + w) & __ldg(D.umask + (size_t)y * P.W + w);
      __syncwarp();
      const float r = spearman_network(D.gem + (size_t)x * P.S, D.gem + (size_t)y * P.S, P.S, mask, buf, lane);
      if ( lane == 0 && B.outCorr ) B.outCorr[q * P.max_k * P.ncorr + (P.corr == 2 ? 1 : 0)] = r;
      __syncwarp();
   }
}

cudaError_t sim_spearman_orders(cudaStream_t st, const DevParams& P, const DevData& D, SpearmanOrders& R)
{
   const int mask = (P.W * 4 + 15) & ~15;
   R.warp_bytes = mask + ((P.S * 2 + 15) & ~15);
   R.net_bytes = mask + 2 * P.P2 * (int)sizeof(float);
   const int smem = P.P2 * (int)sizeof(unsigned long long);
   cudaError_t e = cudaFuncSetAttribute(k_gene_order, cudaFuncAttributeMaxDynamicSharedMemorySize, ORDER_SMEM);
   if ( e == cudaSuccess ) e = cudaFuncSetAttribute(k_spearman_orders, cudaFuncAttributeMaxDynamicSharedMemorySize, SPEARMAN_SMEM);
   if ( e == cudaSuccess ) e = cudaFuncSetAttribute(k_spearman_ties, cudaFuncAttributeMaxDynamicSharedMemorySize, TIES_SMEM);
   if ( e == cudaSuccess )
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&R.per_sm, k_spearman_orders, SPEARMAN_WARPS * 32,
                                                        (size_t)R.warp_bytes * SPEARMAN_WARPS);
   if ( e == cudaSuccess ) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&R.net_per_sm, k_spearman_ties, 32, R.net_bytes);
   if ( e != cudaSuccess ) return e;
   k_gene_order<<<std::min(P.G, 16384), ORDER_THREADS, smem, st>>>(D.gem, D.umask, P.G, P.S, P.W, P.P2, R.order, R.ties);
   return cudaGetLastError();
}

cudaError_t sim_launch_spearman(int sms, cudaStream_t st, const DevParams& P, const DevData& D, const DevBlock& B,
                                const SpearmanOrders& R, int32_t* tied_pairs)
{
   int64_t grid = (int64_t)sms * std::max(1, R.per_sm);
   /* neighbouring pairs share x, so a warp takes up to 8 of them -- fewer if the warps would run out */
   const int per_warp = (int)std::max<int64_t>(1, std::min<int64_t>(8, B.size / (grid * SPEARMAN_WARPS * 4)));
   grid = std::min(grid, (B.size + SPEARMAN_WARPS * per_warp - 1) / (SPEARMAN_WARPS * per_warp));
   k_spearman_orders<<<(int)grid, SPEARMAN_WARPS * 32, R.warp_bytes * SPEARMAN_WARPS, st>>>(P, D, B, R, tied_pairs, R.warp_bytes,
                                                                                            per_warp);
   k_spearman_ties<<<(int)std::min<int64_t>(B.size, (int64_t)sms * std::max(1, R.net_per_sm)), 32, R.net_bytes, st>>>(P, D, B,
                                                                                                             tied_pairs);
   return cudaGetLastError();
}

} /* namespace kinc */
