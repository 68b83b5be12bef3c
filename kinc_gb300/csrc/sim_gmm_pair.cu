/* GMM clustering with one warp per pair (up to 5 components): its launch, and the rule that takes it. */
#include "sim_gmm_pair.cuh"

#include <algorithm>

namespace kinc {

constexpr int GP_SMEM = 227 * 1024 - 16;    /* dynamic shared memory of one CTA: the SM's, beside the kernel's own word */
static int gp_sort_rows(const DevParams& P)
{
   return P.corr >= 1 ? 2 : (P.pre_out || P.post_out) ? 1 : 0;
}

int sim_gmm_pairs_per_sm(const DevParams& P, int n_cap)
{
   if ( P.clus != 1 || P.max_k > GP_KMAX || P.S > 4095 ) return 0;   /* more samples: the pairs' order by N is coarse */
   return GP_SMEM / (gp_slot_floats(std::max(n_cap, 1), P.max_k, gp_sort_rows(P), true) * (int)sizeof(float));
}

/*
 * The tile kernel (one pair per lane) runs whole waves of `wave` pairs, however few there are, and its first wave
 * takes a little longer (10 / n of one, n the usable samples of a pair); this one takes pairs one by one.  It is
 * taken where the block's pairs, in waves, are no more than `rate` times the tile kernel's waves, rate being its own
 * speed against the tile kernel's in full waves: the smaller of two.
 *
 *  - Few samples: the updates between the iterations (123 in units of the tile kernel's sample and component) and
 *    what a sample takes besides its components outweigh the tile kernel's k n.  Measured / this formula, blocks of
 *    389,120 pairs (four waves and 10 / n), Pearson: k <= 2 n = 40: 0.51 / 0.47, 97: 0.79 / 0.77, 243: 1.08 / 1.06;
 *    k <= 3 n = 63: 0.69 / 0.71; k <= 5 n = 40: 0.65 / 0.69, 63: 0.88 / 0.85, 97: 1.04 / 1.00, 162: 1.18 / 1.15.  One cluster
 *    takes two iterations, so the pair's other work decides: n = 40: 0.39 (with outliers and Spearman 0.67), 97:
 *    0.52 (0.88), 243: 0.79 (1.29), 810: 0.93 (1.60), and without sorts at most 0.84 in ten waves.
 *  - Many samples: fewer pairs fit an SM.  97,280 pairs of the 10 %-missing mixture workload, k <= 5, Spearman with
 *    outliers, by pairs that fit: 11 (N = 810) 187k / 168k per second, 8 (N = 1,215) 119k / 113k, 7 (N = 1,620)
 *    81k / 87k, 4 (N = 2,430) 38k / 56k -- about 0.35 + 0.083 per pair.
 */
bool sim_gmm_pairs_better(const DevParams& P, int per_sm, double n, int64_t size, int64_t wave)
{
   if ( per_sm < 1 ) return false;
   n = std::max(n, 1.0);
   double rate;
   if ( P.max_k == 1 )
   {
      rate = gp_sort_rows(P) > 0 ? n / (0.75 * n + 38.0) : std::min(0.82, n / (n + 85.0));
   }
   else
   {
      double tiles = 0.0, here = 0.0;
      for ( int k = std::max(P.min_k, 2); k <= P.max_k; ++k )
      {
         tiles += k * n;
         here += 123.0 + n * (0.16 + 0.62 * k);
      }
      rate = tiles / here;
   }
   rate = std::min(rate, 0.35 + 0.083 * per_sm);
   const double waves = (double)((size + wave - 1) / wave);
   return (double)size / (double)wave <= rate * (waves + 10.0 / n);
}

size_t sim_gmm_pairs_scratch(int sms, const DevParams& P, int n_cap, char* base, DevScratch& W)
{
   const size_t labels = ((size_t)sms * GP_WARPS * P.S + 255) & ~(size_t)255;
   W.lbl = (int8_t*)base;
   W.gam = (float*)(base + labels);
   return labels + (size_t)sms * GP_WARPS * gp_global_floats(n_cap, P.max_k) * sizeof(float);
}

template <int WARPS>
static cudaError_t launch(int sms, cudaStream_t st, const DevParams& P, const DevData& D, const DevScratch& W,
                          const DevBlock& B, int n_cap)
{
   const int rows = gp_sort_rows(P);
   const int slot = gp_slot_floats(std::max(n_cap, 1), P.max_k, rows, false) * (int)sizeof(float);
   const int smem = (int)std::min<int64_t>(GP_SMEM, (int64_t)slot * WARPS);
   const cudaError_t e = cudaFuncSetAttribute(k_gmm_pairs<WARPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, GP_SMEM);
   if ( e != cudaSuccess ) return e;
   const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(B.size, sms));
   k_gmm_pairs<WARPS><<<grid, WARPS * 32, smem, st>>>(P, D, W, B, smem / (int)sizeof(float), rows, n_cap);
   return cudaGetLastError();
}

cudaError_t sim_launch_gmm_pairs(int sms, cudaStream_t st, const DevParams& P, const DevData& D, const DevScratch& W,
                                 const DevBlock& B, int n_cap)
{
   /*
    * 16 warps of 128 registers (the K = 5 fit then reads its E step's parameters per chunk) or 12 of 168, by the
    * pairs an SM holds with vg in shared memory and in global memory; thousands of pairs per second:
    *   N = 122 (15 / 16): 1,030 / 981     N = 243 (12 / 16): 577 / 616
    *   N = 423 (10 / 16): 350 / 303       N = 810 (6 / 11): 174 / 187
    * and 12 where the block gives an SM no more.
    */
   const int rows = gp_sort_rows(P), n = std::max(n_cap, 1);
   const int shared = GP_SMEM / (gp_slot_floats(n, P.max_k, rows, false) * (int)sizeof(float));
   const int global = GP_SMEM / (gp_slot_floats(n, P.max_k, rows, true) * (int)sizeof(float));
   const bool many = B.size > (int64_t)sms * GP_WARPS_FEW && (shared >= 14 || (shared < 11 && global >= 13));
   return many ? launch<GP_WARPS>(sms, st, P, D, W, B, n_cap) : launch<GP_WARPS_FEW>(sms, st, P, D, W, B, n_cap);
}

} /* namespace kinc */
