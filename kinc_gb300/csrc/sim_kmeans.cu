/* K-means: a warp per stream of pairs with register-resident centroids up to K = 3 or 5, the tile kernel with
 * local-memory centroids beyond. */
#include "sim_kmeans_pairs.cuh"

namespace kinc {

SimKernel sim_kernel_kmeans(int max_k)
{
   if ( max_k <= 3 ) return SimKernel { (const void*)&k_kmeans_pairs<3>, 2, 3, false, kernel_warps<2>() };
   if ( max_k <= 5 ) return SimKernel { (const void*)&k_kmeans_pairs<5>, 2, 5, false, kernel_warps<2>() };
   return sim_kernel_handle<2, 0>();
}

cudaError_t sim_launch_kmeans(const SimKernel& k, int grid, int smem, cudaStream_t st, const DevParams& P,
                              const DevData& D, const DevScratch& W, const DevBlock& B, int smem_sort)
{
   switch ( k.ks )
   {
   case 3: k_kmeans_pairs<3><<<grid, P.warps * 32, smem, st>>>(P, D, W, B, smem_sort); break;
   case 5: k_kmeans_pairs<5><<<grid, P.warps * 32, smem, st>>>(P, D, W, B, smem_sort); break;
   default: return sim_kernel_launch<2, 0>(grid, smem, st, P, D, W, B, smem_sort);
   }
   return cudaGetLastError();
}

} /* namespace kinc */
