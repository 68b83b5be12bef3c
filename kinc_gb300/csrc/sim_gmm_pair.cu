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
 * The tile kernel (one pair per lane) runs whole waves of `wave` pairs, however few there are; this one
 * takes pairs one by one.  Their rates at full waves, 97,280 pairs of the 10 %-missing mixture workload,
 * this kernel / the tile kernel, by pairs that fit an SM: 11 (N = 810) 187k / 168k per second, 10
 * (N = 1,134) 127k / 118k, 7 (N = 1,620) 81k / 87k, 4 (N = 2,430) 38k / 56k -- about 0.35 + 0.083 per
 * pair.  The tile kernel is taken where its wave is fuller than that.
 */
bool sim_gmm_pairs_better(int per_sm, int64_t size, int64_t wave)
{
   if ( per_sm < 1 ) return false;
   const double full = (double)size / (double)((size + wave - 1) / wave * wave);
   return full <= 0.35 + 0.083 * per_sm;
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
