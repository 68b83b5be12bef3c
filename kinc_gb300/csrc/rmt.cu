/*
 * rmt.cu -- the RMT analytic (include/kinc_rmt.h).
 *
 * GPU: per-(gene, cluster) largest |r| from the CMX items (computeMaximums,
 * src/core/rmt.cpp:164-195), then per threshold the connected components of
 * the pruned matrix (computePruneMatrix, :202-245), each scattered straight
 * from the items into a dense double array in HBM, and their eigenvalues
 * (computeEigenvalues, :252-282, which solves the same double matrix): one
 * kernel for all components of up to 128 rows, cuSOLVER's symmetric
 * divide-and-conquer solver for larger ones, or for all rows together where that
 * costs no more (rmt_plan).
 *
 * Host: the eigenvalues sorted by ascending |lambda| and converted to float,
 * the unique values (degenerate, :374-388), the Akima-spline unfolding
 * (unfold, :395-439) and the chi-square against the Poisson spacing
 * distribution averaged over unfolding paces (computeChiSquare /
 * computePaceChiSquare, :289-367), in the reference's float/double types.
 * The reference calls GSL for the spline (gsl_interp_akima; GSL is not part
 * of the KINC tree and no version is pinned): the spline here is Akima's
 * published method (H. Akima, J. ACM 17(4), 1970) with the usual end
 * extension of the slopes, written from that description.
 */
#include "../../include/kinc_rmt.h"
#include "../../include/kinc_pairwise_matrix.h"
#include "kinc_fmath.h"

#include <cuda_runtime.h>
#include <cusolverDn.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <limits>
#include <string>
#include <vector>

namespace {

thread_local std::string r_err;

int rmt_fail(int code, const char* fmt, ...)
{
   char buf[512];
   va_list ap;
   va_start(ap, fmt);
   vsnprintf(buf, sizeof buf, fmt, ap);
   va_end(ap);
   r_err = buf;
   return code;
}

/* ------------------------------------------------------------------ GPU */

/* largest |r| per (gene, cluster); |r| >= 0 so its bits order like the value; NaN never wins */
__global__ void k_rmt_max(int64_t n, int K, const int32_t* __restrict__ x, const int32_t* __restrict__ y,
                          const int8_t* __restrict__ c, const float* __restrict__ r, unsigned int* __restrict__ mx)
{
   for ( int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x )
   {
      const float a = fabsf(r[i]);
      if ( !(a == a) ) continue;
      atomicMax(&mx[(int64_t)x[i] * K + c[i]], __float_as_uint(a));
      atomicMax(&mx[(int64_t)y[i] * K + c[i]], __float_as_uint(a));
   }
}

/*
 * Components.  The pruned matrix joins two rows only where an item is kept, and at the thresholds of a search most
 * rows sit in small groups; after a permutation the matrix is block diagonal, and its eigenvalues are the blocks'.
 * So the rows are united along the kept items, components of up to RMT_BLOCK rows are solved by k_rmt_blocks, all in
 * one launch, and only larger ones go to cuSOLVER (rmt_plan: also where the whole matrix in one solve is faster).  A 1,000-row matrix of 10-row components:
 * 23.5 -> 0.7 ms; a search over 50 thresholds of 5,000 rows in 5-row components 10.5 -> 0.1 s.
 */
constexpr int RMT_BLOCK = 128;              /* rows of a block k_rmt_blocks holds in shared memory (128 KB) */
constexpr int RMT_BLOCK_WARP = 32;          /* up to this many, one warp per block */

/* kept rows start as their own root, the others as -1 */
__global__ void k_rmt_roots(int64_t rows, const unsigned int* __restrict__ mx, float t, int32_t* __restrict__ root)
{
   for ( int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < rows; i += (int64_t)gridDim.x * blockDim.x )
      root[i] = __uint_as_float(mx[i]) >= t ? (int32_t)i : -1;
}

/* The root of i, halving the path on the way (a root's parent is itself, any other's is smaller).  Union-find with
 * path halving and roots hung by compare-and-swap: R. J. Anderson, H. Woll, Wait-free parallel algorithms for the
 * union-find problem, STOC 1991. */
__device__ __forceinline__ int32_t rmt_find(volatile int32_t* root, int32_t i)
{
   int32_t p = root[i];
   while ( p != i )
   {
      const int32_t g = root[p];
      if ( g != p ) root[i] = g;
      i = p;
      p = g;
   }
   return i;
}

/* unites the rows of every kept item: the larger root is hung below the smaller one */
__global__ void k_rmt_unite(int64_t n, int K, const int32_t* __restrict__ x, const int32_t* __restrict__ y,
                            const int8_t* __restrict__ c, const float* __restrict__ r, float t, int32_t* root)
{
   for ( int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x )
   {
      if ( !(fabsf(r[i]) >= t) ) continue;
      int32_t a = rmt_find(root, x[i] * K + c[i]), b = rmt_find(root, y[i] * K + c[i]);
      while ( a != b )
      {
         if ( a < b )
         {
            const int32_t s = a;
            a = b;
            b = s;
         }
         /* roots only ever get smaller, so every failed exchange moves a down: the loop ends */
         const int32_t was = atomicCAS(&root[a], a, b);
         if ( was == a ) break;
         a = rmt_find(root, was);
         b = rmt_find(root, b);
      }
   }
}

/* every kept row's root.  No halving here: each entry has one writer, so what is left in it is the root (a
 * neighbour's halving could put an older ancestor back). */
__global__ void k_rmt_flatten(int64_t rows, int32_t* root)
{
   volatile const int32_t* parent = root;
   for ( int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < rows; i += (int64_t)gridDim.x * blockDim.x )
   {
      int32_t p = parent[i];
      if ( p < 0 ) continue;
      for ( int32_t g = parent[p]; g != p; g = parent[p] ) p = g;
      root[i] = p;
   }
}

/* a matrix to solve (one component or several): its rows, and where it (row-major, lower triangle) and its eigenvalues
 * lie */
struct RmtComponent
{
   int64_t at;
   int32_t size, values;
};

/* the unit diagonals and the kept items; place[row] = { matrix, position in it } */
__global__ void k_rmt_fill(int64_t rows, int64_t n, int K, const int32_t* __restrict__ x, const int32_t* __restrict__ y,
                           const int8_t* __restrict__ c, const float* __restrict__ r, float t,
                           const int2* __restrict__ place, const RmtComponent* __restrict__ comp, double* __restrict__ A)
{
   for ( int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < rows + n; i += (int64_t)gridDim.x * blockDim.x )
   {
      if ( i < rows )
      {
         const int2 p = place[i];
         if ( p.x >= 0 ) A[comp[p.x].at + (int64_t)p.y * (comp[p.x].size + 1)] = 1.0;
         continue;
      }
      const int64_t k = i - rows;
      const float v = r[k];
      if ( !(fabsf(v) >= t) ) continue;
      const int2 a = place[(int64_t)x[k] * K + c[k]], b = place[(int64_t)y[k] * K + c[k]];
      if ( a.x < 0 || a.x != b.x ) continue;
      A[comp[a.x].at + (int64_t)a.y * comp[a.x].size + b.y] = (double)v;
   }
}

/* sum over the CTA; every thread gets it (red: 32 doubles of shared memory) */
__device__ __forceinline__ double rmt_sum(double v, double* red)
{
   for ( int o = 16; o > 0; o >>= 1 ) v += __shfl_xor_sync(0xffffffffu, v, o);
   if ( blockDim.x == 32 ) return v;
   __syncthreads();
   if ( (threadIdx.x & 31) == 0 ) red[threadIdx.x >> 5] = v;
   __syncthreads();
   double s = 0.0;
   for ( int i = 0; i < (int)(blockDim.x >> 5); ++i ) s += red[i];
   return s;
}

/*
 * Eigenvalues of one component per CTA, in double: Householder reduction to tridiagonal form in shared memory, then
 * every eigenvalue by bisection on the count of negative pivots (Sturm's theorem; W. Barth, R. S. Martin, J. H.
 * Wilkinson, Numer. Math. 9, 1967), one thread each.  Bound by the latency of FP64 divisions, of which a bisection step
 * makes one per row.
 */
__global__ void k_rmt_blocks(const RmtComponent* __restrict__ comp, const int32_t* __restrict__ list, int count,
                             const double* __restrict__ A, double* __restrict__ W)
{
   extern __shared__ double rmt_smem[];
   if ( (int)blockIdx.x >= count ) return;
   const RmtComponent q = comp[list[blockIdx.x]];
   const int n = q.size, ld = n + 1, tid = threadIdx.x;
   double* M = rmt_smem;                     /* [n][ld], both triangles */
   double* d = M + n * ld;
   double* e = d + n;                        /* e[i]: between rows i and i + 1, squared later */
   double* v = e + n;
   double* w = v + n;
   double* red = w + n;
   for ( int i = tid; i < n * n; i += blockDim.x )
   {
      const int row = i / n, col = i % n;
      const double a = col <= row ? A[q.at + (int64_t)row * n + col] : A[q.at + (int64_t)col * n + row];
      M[row * ld + col] = a;
   }
   __syncthreads();
   for ( int k = 0; k + 1 < n; ++k )
   {
      /* column k below the diagonal onto its first element */
      double s = 0.0;
      for ( int i = k + 2 + tid; i < n; i += blockDim.x ) s += M[i * ld + k] * M[i * ld + k];
      s = rmt_sum(s, red);
      const double x0 = M[(k + 1) * ld + k];
      if ( tid == 0 ) d[k] = M[k * ld + k];
      if ( s == 0.0 )
      {
         if ( tid == 0 ) e[k] = x0;
         __syncthreads();
         continue;
      }
      const double norm = sqrt(x0 * x0 + s), alpha = x0 > 0.0 ? -norm : norm, v0 = x0 - alpha;
      const double beta = 2.0 / (v0 * v0 + s);
      if ( tid == 0 ) e[k] = alpha;
      for ( int i = k + 1 + tid; i < n; i += blockDim.x ) v[i] = i == k + 1 ? v0 : M[i * ld + k];
      __syncthreads();
      /* w = beta M v - (beta / 2) (v, beta M v) v */
      double dot = 0.0;
      for ( int i = k + 1 + tid; i < n; i += blockDim.x )
      {
         double p = 0.0;
         for ( int j = k + 1; j < n; ++j ) p += M[j * ld + i] * v[j];
         p *= beta;
         w[i] = p;
         dot += p * v[i];
      }
      dot = 0.5 * beta * rmt_sum(dot, red);
      for ( int i = k + 1 + tid; i < n; i += blockDim.x ) w[i] -= dot * v[i];
      __syncthreads();
      for ( int i = k + 1 + tid; i < n; i += blockDim.x )
      {
         const double vi = v[i], wi = w[i];
         for ( int j = k + 1; j < n; ++j ) M[j * ld + i] -= v[j] * wi + w[j] * vi;
      }
      __syncthreads();
   }
   if ( tid == 0 )
   {
      d[n - 1] = M[(n - 1) * ld + n - 1];
      e[n - 1] = 0.0;
   }
   __syncthreads();
   /* Gershgorin's bounds, with room for the reduction's rounding */
   double lo = 1e300, hi = -1e300;
   for ( int i = 0; i < n; ++i )
   {
      const double r = (i > 0 ? fabs(e[i - 1]) : 0.0) + fabs(e[i]);
      lo = fmin(lo, d[i] - r);
      hi = fmax(hi, d[i] + r);
   }
   const double span = fmax(fabs(lo), fabs(hi)), tiny = span * 1e-30;
   lo -= span * 1e-14;
   hi += span * 1e-14;
   for ( int j = tid; j < n; j += blockDim.x )
   {
      /* the j-th smallest: at most j eigenvalues below a, more than j below b */
      double a = lo, b = hi;
      for ( int it = 0; it < 80; ++it )
      {
         const double x = 0.5 * (a + b);
         if ( x <= a || x >= b ) break;
         int below = 0;
         double p = 1.0;
         for ( int i = 0; i < n; ++i )
         {
            const double ee = i > 0 ? e[i - 1] * e[i - 1] : 0.0;
            p = d[i] - x - ee / p;
            if ( fabs(p) < tiny ) p = -tiny;
            below += p < 0.0;
         }
         if ( below > j )
            b = x;
         else
            a = x;
         if ( b - a <= 1e-16 * span ) break;
      }
      W[q.values + j] = 0.5 * (a + b);
   }
}

static size_t rmt_block_bytes(int n)
{
   return ((size_t)n * (n + 1) + 4 * (size_t)n + 32) * sizeof(double);
}

struct RmtDevice
{
   int32_t G = 0, K = 0;
   int64_t n = 0;
   int sms = 1;
   bool infinite = false;              /* an item is infinite */
   int32_t *dx = nullptr, *dy = nullptr, *droot = nullptr, *dlist = nullptr, *dinfo = nullptr;
   int2* dplace = nullptr;
   RmtComponent* dcomp = nullptr;
   std::vector<int32_t> root;          /* host copies, kept for their room */
   std::vector<int2> place;
   int8_t* dc = nullptr;
   float* dr = nullptr;
   unsigned int* dmax = nullptr;
   double *dA = nullptr, *dW = nullptr, *dwork = nullptr;
   size_t capA = 0, capWork = 0;
   cudaStream_t st = nullptr;
   cusolverDnHandle_t solver = nullptr;

   ~RmtDevice()
   {
      cudaFree(dx); cudaFree(dy); cudaFree(droot); cudaFree(dlist); cudaFree(dinfo); cudaFree(dplace); cudaFree(dcomp); cudaFree(dc); cudaFree(dr);
      cudaFree(dmax); cudaFree(dA); cudaFree(dW); cudaFree(dwork);
      if ( solver ) cusolverDnDestroy(solver);
      if ( st ) cudaStreamDestroy(st);
   }
};

#define RCK(call)                                                                                  \
   do                                                                                              \
   {                                                                                               \
      cudaError_t e_ = (call);                                                                     \
      if ( e_ != cudaSuccess )                                                                     \
         return rmt_fail(e_ == cudaErrorMemoryAllocation ? KINC_SIM_ENOMEM : KINC_SIM_ECUDA, "%s: %s", \
                         #call, cudaGetErrorString(e_));                                           \
   } while ( 0 )

int device_setup(RmtDevice& d, int32_t G, int32_t K, int64_t n, const int32_t* x, const int32_t* y, const int8_t* c,
                 const float* r)
{
   if ( G < 1 || K < 1 || n < 0 || (n > 0 && (!x || !y || !c || !r)) )
      return rmt_fail(KINC_SIM_EINVAL, "Did not get valid input or logfile arguments.");
   for ( int64_t i = 0; i < n; ++i )
      if ( x[i] <= y[i] || y[i] < 0 || x[i] >= G || c[i] < 0 || c[i] >= K )
         return rmt_fail(KINC_SIM_EINVAL, "item %lld (%d, %d, %d) outside %d genes x %d clusters", (long long)i, x[i],
                         y[i], c[i], G, K);
   int infinite = 0;                                     /* no early end: this loop is vectorised */
   for ( int64_t i = 0; i < n; ++i ) infinite |= std::fabs(r[i]) > std::numeric_limits<float>::max();
   d.infinite = infinite != 0;
   d.G = G;
   d.K = K;
   d.n = n;
   const int64_t rows = (int64_t)G * K;
   int dev = 0;
   RCK(cudaGetDevice(&dev));
   RCK(cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev));
   RCK(cudaStreamCreateWithFlags(&d.st, cudaStreamNonBlocking));
   RCK(cudaMalloc(&d.dx, std::max<int64_t>(n, 1) * 4));
   RCK(cudaMalloc(&d.dy, std::max<int64_t>(n, 1) * 4));
   RCK(cudaMalloc(&d.dc, std::max<int64_t>(n, 1)));
   RCK(cudaMalloc(&d.dr, std::max<int64_t>(n, 1) * 4));
   RCK(cudaMalloc(&d.dmax, rows * sizeof(unsigned int)));
   RCK(cudaMalloc(&d.droot, rows * sizeof(int32_t)));
   RCK(cudaMalloc(&d.dlist, rows * sizeof(int32_t)));
   RCK(cudaMalloc(&d.dplace, rows * sizeof(int2)));
   RCK(cudaMalloc(&d.dcomp, rows * sizeof(RmtComponent)));
   RCK(cudaMalloc(&d.dW, rows * sizeof(double)));
   if ( n > 0 )
   {
      RCK(cudaMemcpyAsync(d.dx, x, n * 4, cudaMemcpyHostToDevice, d.st));
      RCK(cudaMemcpyAsync(d.dy, y, n * 4, cudaMemcpyHostToDevice, d.st));
      RCK(cudaMemcpyAsync(d.dc, c, n, cudaMemcpyHostToDevice, d.st));
      RCK(cudaMemcpyAsync(d.dr, r, n * 4, cudaMemcpyHostToDevice, d.st));
   }
   RCK(cudaMemsetAsync(d.dmax, 0, rows * sizeof(unsigned int), d.st));   /* the reference starts every maximum at 0 */
   if ( n > 0 )
   {
      const int blocks = (int)std::min<int64_t>((n + 255) / 256, 4096);
      k_rmt_max<<<blocks, 256, 0, d.st>>>(n, K, d.dx, d.dy, d.dc, d.dr, d.dmax);
      RCK(cudaGetLastError());
   }
   return KINC_SIM_OK;
}

/*
 * Which matrices the components are solved in.  into[k] = { matrix, first row in it } of component k; the sizes of the
 * matrices are returned.  Those of up to RMT_BLOCK rows run in k_rmt_blocks if `blocks` is set on return.
 *
 * Times of one threshold, in the 0.030 ms that the library's solver takes per row: a matrix of r rows max(r, r^2 / 1,700)
 * there (64 rows 1.6 ms, 128 4.1, 200 6.0, 1,000 30, 3,000 159, 7,800 1,063), and k_rmt_blocks 1.5 per row of its largest
 * component, whatever their number up to a wave (32 rows 1.3 ms, 64 2.6, 128 6.1; 10 of 128 6.2).  So
 *  - one matrix of all rows where that is no slower than the parts: one component with two thirds of the rows or more
 *    (a component of 64 rows alone: 2.6 -> 1.6 ms);
 *  - else the components above RMT_BLOCK rows share matrices of about RMT_SHARED rows, up to which a row costs the same
 *    and each solve by itself costs more (8 components of 129 rows: 34.5 -> 27.5 ms).
 */
constexpr double RMT_SHARED = 1280.0;

static std::vector<int32_t> rmt_plan(const std::vector<int32_t>& size, int sms, std::vector<int2>& into, bool& blocks)
{
   auto solver = [](double r) { return std::max(r, r * r / 1700.0); };
   double all = 0.0, large = 0.0;
   int32_t most[2] = { 0, 0 };
   int64_t count[2] = { 0, 0 };
   for ( int32_t n : size )
   {
      all += n;
      if ( n > RMT_BLOCK )
         large += n;
      else
      {
         const int wide = n > RMT_BLOCK_WARP;
         most[wide] = std::max(most[wide], n);
         ++count[wide];
      }
   }
   const int groups = (int)std::ceil(large / RMT_SHARED);
   const double target = groups > 0 ? large / groups : 0.0;
   std::vector<int32_t> matrix;
   into.assign(size.size(), make_int2(0, 0));
   double parts = 0.0;
   int shared = -1;                                      /* the matrix that large components are being added to */
   for ( size_t k = 0; k < size.size(); ++k )
   {
      if ( size[k] <= RMT_BLOCK || shared < 0 || matrix[(size_t)shared] >= target )
      {
         into[k] = make_int2((int)matrix.size(), 0);
         if ( size[k] > RMT_BLOCK ) shared = (int)matrix.size();
         matrix.push_back(size[k]);
      }
      else
      {
         into[k] = make_int2(shared, matrix[(size_t)shared]);
         matrix[(size_t)shared] += size[k];
      }
   }
   for ( int32_t n : matrix )
      if ( n > RMT_BLOCK ) parts += solver(n);
   for ( int wide = 0; wide < 2; ++wide )
   {
      const double per_sm = std::min(32.0, std::floor(227.0 * 1024 / (double)(rmt_block_bytes(most[wide]) + 1024)));
      parts += 1.5 * most[wide] * std::ceil((double)count[wide] / (per_sm * sms));
   }
   blocks = solver(all) > parts;
   if ( !blocks )
   {
      int32_t at = 0;
      for ( size_t k = 0; k < size.size(); ++k )
      {
         into[k] = make_int2(0, at);
         at += size[k];
      }
      matrix.assign(1, at);
   }
   return matrix;
}

/* the eigenvalues of one matrix by the library: from dA + at into dW + values */
int large_matrix(RmtDevice& d, const RmtComponent& q)
{
   if ( !d.solver && (cusolverDnCreate(&d.solver) != CUSOLVER_STATUS_SUCCESS
                      || cusolverDnSetStream(d.solver, d.st) != CUSOLVER_STATUS_SUCCESS) )
      return rmt_fail(KINC_SIM_ECUDA, "cannot create the eigensolver");
   if ( !d.dinfo ) RCK(cudaMalloc(&d.dinfo, sizeof(int32_t)));
   /* row-major with the lower triangle set = column-major with the upper triangle set */
   const int32_t m = q.size;
   double* A = d.dA + q.at;
   int lwork = 0;
   if ( cusolverDnDsyevd_bufferSize(d.solver, CUSOLVER_EIG_MODE_NOVECTOR, CUBLAS_FILL_MODE_UPPER, m, A, m, d.dW + q.values,
                                    &lwork) != CUSOLVER_STATUS_SUCCESS )
      return rmt_fail(KINC_SIM_ECUDA, "eigensolver workspace query failed for m = %d", m);
   if ( (size_t)lwork > d.capWork )
   {
      cudaFree(d.dwork);
      d.dwork = nullptr;
      d.capWork = 0;
      RCK(cudaMalloc(&d.dwork, (size_t)lwork * sizeof(double)));
      d.capWork = (size_t)lwork;
   }
   if ( cusolverDnDsyevd(d.solver, CUSOLVER_EIG_MODE_NOVECTOR, CUBLAS_FILL_MODE_UPPER, m, A, m, d.dW + q.values, d.dwork,
                         lwork, d.dinfo) != CUSOLVER_STATUS_SUCCESS )
      return rmt_fail(KINC_SIM_ECUDA, "eigensolver failed for m = %d", m);
   int32_t info = 0;
   RCK(cudaMemcpyAsync(&info, d.dinfo, sizeof(int32_t), cudaMemcpyDeviceToHost, d.st));
   RCK(cudaStreamSynchronize(d.st));
   if ( info != 0 ) return rmt_fail(KINC_SIM_ECUDA, "eigensolver did not converge (info %d, m = %d)", info, m);
   return KINC_SIM_OK;
}

/* eigenvalues of the pruned matrix at threshold t, ascending |lambda|, as floats */
int device_eigenvalues(RmtDevice& d, float t, std::vector<float>& eig, int32_t& m)
{
   const int64_t rows = (int64_t)d.G * d.K;
   const int by_row = (int)std::min<int64_t>((rows + 255) / 256, 4096), by_item = (int)std::min<int64_t>((d.n + 255) / 256, 4096);
   k_rmt_roots<<<by_row, 256, 0, d.st>>>(rows, d.dmax, t, d.droot);
   if ( d.n > 0 ) k_rmt_unite<<<by_item, 256, 0, d.st>>>(d.n, d.K, d.dx, d.dy, d.dc, d.dr, t, d.droot);
   k_rmt_flatten<<<by_row, 256, 0, d.st>>>(rows, d.droot);
   RCK(cudaGetLastError());
   d.root.resize((size_t)rows);
   d.place.resize((size_t)rows);
   RCK(cudaMemcpyAsync(d.root.data(), d.droot, (size_t)rows * sizeof(int32_t), cudaMemcpyDeviceToHost, d.st));
   RCK(cudaStreamSynchronize(d.st));

   /* the components in the order of their first rows, and each row's place */
   eig.clear();
   m = 0;
   std::vector<int32_t> size;
   for ( int64_t i = 0; i < rows; ++i )
   {
      const int32_t root = d.root[(size_t)i];
      int2 p = make_int2(-1, 0);
      if ( root >= 0 )
      {
         if ( root == i )
         {
            p.x = (int)size.size();
            size.push_back(0);
         }
         else
            p.x = d.place[(size_t)root].x;               /* a root is its component's first row */
         p.y = size[(size_t)p.x]++;
         ++m;
      }
      d.place[(size_t)i] = p;
   }
   if ( m == 0 ) return KINC_SIM_OK;
   if ( d.infinite )
   {
      /* every threshold keeps an infinite item, and a matrix with one has no eigenvalues.  The reference's dense
       * solver turns all that it meets afterwards into NaN; here none are computed: bisection would return finite
       * values (fmin and fmax drop the NaN that the reduction makes of an infinity) */
      eig.assign((size_t)m, std::numeric_limits<float>::quiet_NaN());
      return KINC_SIM_OK;
   }
   std::vector<int2> into;
   bool blocks = true;
   const std::vector<int32_t> matrix = rmt_plan(size, d.sms, into, blocks);
   if ( matrix.size() != size.size() )
      for ( int2& p : d.place )
         if ( p.x >= 0 ) p = make_int2(into[(size_t)p.x].x, into[(size_t)p.x].y + p.y);
   auto in_block = [&](int32_t n) { return blocks && n <= RMT_BLOCK; };
   size_t need = 0;
   int32_t values = 0, most[2] = { 0, 0 };
   std::vector<RmtComponent> comp;
   std::vector<int32_t> list[2];                         /* blocks for a warp, and for a larger CTA */
   for ( int32_t n : matrix )
   {
      if ( !in_block(n) ) need = (need + 31) & ~(size_t)31;      /* the library's matrices on 256-byte boundaries */
      comp.push_back(RmtComponent { (int64_t)need, n, values });
      need += (size_t)n * n;
      values += n;
      if ( !in_block(n) ) continue;
      const int wide = n > RMT_BLOCK_WARP;
      list[wide].push_back((int32_t)comp.size() - 1);
      most[wide] = std::max(most[wide], n);
   }
   if ( need > d.capA )
   {
      cudaFree(d.dA);
      d.dA = nullptr;
      d.capA = 0;
      RCK(cudaMalloc(&d.dA, need * sizeof(double)));
      d.capA = need;
   }
   RCK(cudaMemsetAsync(d.dA, 0, need * sizeof(double), d.st));
   RCK(cudaMemcpyAsync(d.dplace, d.place.data(), (size_t)rows * sizeof(int2), cudaMemcpyHostToDevice, d.st));
   RCK(cudaMemcpyAsync(d.dcomp, comp.data(), comp.size() * sizeof(RmtComponent), cudaMemcpyHostToDevice, d.st));
   k_rmt_fill<<<(int)std::min<int64_t>((rows + d.n + 255) / 256, 4096), 256, 0, d.st>>>(rows, d.n, d.K, d.dx, d.dy, d.dc, d.dr,
                                                                                        t, d.dplace, d.dcomp, d.dA);
   RCK(cudaGetLastError());
   int32_t* to = d.dlist;
   for ( int wide = 0; wide < 2; ++wide )
   {
      const int count = (int)list[wide].size();
      if ( count == 0 ) continue;
      const int smem = (int)rmt_block_bytes(most[wide]);
      RCK(cudaMemcpyAsync(to, list[wide].data(), (size_t)count * sizeof(int32_t), cudaMemcpyHostToDevice, d.st));
      /* the kernel's limit, the same for every caller (it belongs to the kernel, not to a call) */
      if ( smem > 48 * 1024 )
         RCK(cudaFuncSetAttribute(k_rmt_blocks, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rmt_block_bytes(RMT_BLOCK)));
      k_rmt_blocks<<<count, wide ? RMT_BLOCK : RMT_BLOCK_WARP, smem, d.st>>>(d.dcomp, to, count, d.dA, d.dW);
      RCK(cudaGetLastError());
      to += count;
   }
   for ( const RmtComponent& q : comp )
   {
      if ( in_block(q.size) ) continue;
      const int rc = large_matrix(d, q);
      if ( rc ) return rc;
   }
   std::vector<double> w((size_t)m);
   RCK(cudaMemcpyAsync(w.data(), d.dW, (size_t)m * sizeof(double), cudaMemcpyDeviceToHost, d.st));
   RCK(cudaStreamSynchronize(d.st));
   /* GSL_EIGEN_SORT_ABS_ASC: ascending |lambda| (ascending among equal magnitudes); a NaN would come last */
   std::sort(w.begin(), w.end(), [](double a, double b) {
      if ( std::isnan(a) || std::isnan(b) ) return !std::isnan(a) && std::isnan(b);
      const double fa = std::fabs(a), fb = std::fabs(b);
      return fa != fb ? fa < fb : a < b;
   });
   eig.resize((size_t)m);
   for ( int32_t i = 0; i < m; ++i ) eig[(size_t)i] = (float)w[(size_t)i];
   return KINC_SIM_OK;
}

/* ----------------------------------------------------------------- host */

/* Akima spline through (x[i], y[i]), x strictly increasing, n >= 5 */
struct Akima
{
   std::vector<double> x, y, b, c, d;

   bool init(const double* xs, const double* ys, int n)
   {
      x.assign(xs, xs + n);
      y.assign(ys, ys + n);
      for ( int i = 0; i + 1 < n; ++i )
         if ( !(x[(size_t)i] < x[(size_t)i + 1]) ) return false;
      /* slopes m[-2 .. n] stored at m[j + 2] */
      std::vector<double> m((size_t)n + 3);
      for ( int i = 0; i + 1 < n; ++i )
         m[(size_t)i + 2] = (y[(size_t)i + 1] - y[(size_t)i]) / (x[(size_t)i + 1] - x[(size_t)i]);
      m[1] = 2.0 * m[2] - m[3];
      m[0] = 3.0 * m[2] - 2.0 * m[3];
      m[(size_t)n + 1] = 2.0 * m[(size_t)n] - m[(size_t)n - 1];
      m[(size_t)n + 2] = 3.0 * m[(size_t)n] - 2.0 * m[(size_t)n - 1];
      auto M = [&](int j) { return m[(size_t)(j + 2)]; };
      /* derivative at each knot: weights from the slope differences on either side */
      std::vector<double> tk((size_t)n);
      for ( int i = 0; i < n; ++i )
      {
         const double w1 = std::fabs(M(i + 1) - M(i));
         const double w2 = std::fabs(M(i - 1) - M(i - 2));
         const double ne = w1 + w2;
         if ( ne == 0.0 )
         {
            tk[(size_t)i] = 0.5 * (M(i - 1) + M(i));
         }
         else
         {
            const double alpha = w2 / ne;
            tk[(size_t)i] = (1.0 - alpha) * M(i - 1) + alpha * M(i);
         }
      }
      b.assign((size_t)n, 0.0);
      c.assign((size_t)n, 0.0);
      d.assign((size_t)n, 0.0);
      for ( int i = 0; i + 1 < n; ++i )
      {
         const double h = x[(size_t)i + 1] - x[(size_t)i];
         b[(size_t)i] = tk[(size_t)i];
         c[(size_t)i] = (3.0 * M(i) - 2.0 * tk[(size_t)i] - tk[(size_t)i + 1]) / h;
         d[(size_t)i] = (tk[(size_t)i] + tk[(size_t)i + 1] - 2.0 * M(i)) / (h * h);
      }
      return true;
   }

   double eval(double v) const
   {
      /* interval i with x[i] <= v < x[i+1]; v == x[n-1] takes the last interval */
      const int n = (int)x.size();
      int lo = 0, hi = n - 1;
      while ( hi - lo > 1 )
      {
         const int mid = (lo + hi) / 2;
         if ( x[(size_t)mid] > v ) hi = mid; else lo = mid;
      }
      const double dx = v - x[(size_t)lo];
      return y[(size_t)lo] + dx * (b[(size_t)lo] + dx * (c[(size_t)lo] + dx * d[(size_t)lo]));
   }
};

/* unique eigenvalues: skips the first, drops values within 1e-6 of the last kept (degenerate) */
std::vector<float> unique_eigens(const float* e, int n)
{
   const float EPSILON = 1e-6f;
   std::vector<float> u;
   for ( int i = 1; i < n; ++i )
      if ( u.empty() || std::fabs(e[i] - u.back()) > EPSILON ) u.push_back(e[i]);
   return u;
}

/* unfold: spacings of the spline-unfolded eigenvalues; false when the spline rejects the knots */
bool unfold(const std::vector<float>& e, int pace, std::vector<float>& spacings)
{
   const int n = (int)e.size();
   const int ns = n / pace;
   std::vector<double> x((size_t)ns), y((size_t)ns);
   for ( int i = 0; i < ns; ++i )
   {
      x[(size_t)i] = (double)e[(size_t)i * pace];
      y[(size_t)i] = (double)(i * pace + 1) / n;
   }
   x[(size_t)ns - 1] = e.back();
   y[(size_t)ns - 1] = 1.0;
   Akima s;
   if ( !s.init(x.data(), y.data(), ns) ) return false;
   std::vector<float> se((size_t)n);
   se[0] = 0.0f;
   se[(size_t)n - 1] = 1.0f;
   for ( int i = 1; i < n - 1; ++i )
   {
      const double v = (double)e[(size_t)i];
      if ( v < x.front() || v > x.back() ) return false;   /* outside the spline's range */
      se[(size_t)i] = (float)s.eval(v);
   }
   spacings.resize((size_t)n - 1);
   for ( int i = 0; i < n - 1; ++i ) spacings[(size_t)i] = (se[(size_t)i + 1] - se[(size_t)i]) * n;
   return true;
}

/* computePaceChiSquare: NNSD histogram on [0, 3) against the Poisson spacing law */
bool pace_chi(const std::vector<float>& e, int pace, int bins, float& chi)
{
   std::vector<float> sp;
   if ( !unfold(e, pace, sp) ) return false;
   const float hmin = 0.0f, hmax = 3.0f;
   const float w = (hmax - hmin) / bins;
   std::vector<float> hist((size_t)bins, 0.0f);
   for ( float s : sp )
   {
      if ( hmin <= s && s < hmax )
      {
         const int b = (int)((s - hmin) / w);
         if ( b < bins ) ++hist[(size_t)b];   /* a spacing just below 3 can round into bin `bins` */
      }
   }
   chi = 0.0f;
   const int n = (int)e.size();
   for ( int i = 0; i < bins; ++i )
   {
      const float O = hist[(size_t)i];
      const float E = (kinc_expf(-i * w) - kinc_expf(-(i + 1) * w)) * n;
      chi += (O - E) * (O - E) / E;
   }
   return true;
}

int chi_square(const float* eigens, int n, const kinc_rmt_params& p, float& chi)
{
   const std::vector<float> u = unique_eigens(eigens, n);
   if ( (int)u.size() < p.min_eigenvalue_size )
   {
      chi = -1.0f;
      return KINC_SIM_OK;
   }
   chi = 0.0f;
   int count = 0;
   for ( int pace = p.min_unfolding_pace; pace <= p.max_unfolding_pace; ++pace )
   {
      if ( (int)u.size() / pace < 5 ) break;
      float c = 0.0f;
      if ( !pace_chi(u, pace, p.histogram_bin_size, c) )
         return rmt_fail(KINC_RMT_ESPLINE, "unfolding at pace %d: eigenvalues not increasing in |lambda| order", pace);
      chi += c;
      ++count;
   }
   chi /= count;
   return KINC_SIM_OK;
}

int check_params(const kinc_rmt_params* p)
{
   if ( !p ) return rmt_fail(KINC_SIM_EINVAL, "no parameters");
   if ( p->threshold_start <= p->threshold_stop )
      return rmt_fail(KINC_SIM_EINVAL, "Starting threshold must be greater than stopping threshold.");
   if ( p->min_unfolding_pace >= p->max_unfolding_pace )
      return rmt_fail(KINC_SIM_EINVAL, "Minimum unfolding pace must be less than maximum unfolding pace.");
   if ( p->min_unfolding_pace < 1 || p->histogram_bin_size < 1 || !(p->threshold_step > 0.0f) )
      return rmt_fail(KINC_SIM_EINVAL, "An integer argument given is less than the minimum.");
   return KINC_SIM_OK;
}

}  // namespace

extern "C" void kinc_rmt_params_default(kinc_rmt_params* p)
{
   if ( !p ) return;
   p->threshold_start = 0.99f;
   p->threshold_step = 0.001f;
   p->threshold_stop = 0.5f;
   p->chi_square_threshold1 = 99.607f;
   p->chi_square_threshold2 = 200.0f;
   p->min_eigenvalue_size = 50;
   p->min_unfolding_pace = 10;
   p->max_unfolding_pace = 40;
   p->histogram_bin_size = 60;
}

extern "C" const char* kinc_rmt_last_error(void)
{
   return r_err.c_str();
}

extern "C" int kinc_rmt_chi_square(const float* eigens, int32_t n, const kinc_rmt_params* p, float* out_chi)
{
   if ( !out_chi || n < 0 || (n > 0 && !eigens) ) return rmt_fail(KINC_SIM_EINVAL, "invalid arguments");
   int rc = check_params(p);
   if ( rc ) return rc;
   return chi_square(eigens, n, *p, *out_chi);
}

extern "C" int kinc_rmt_prune_eigenvalues(int32_t genes, int32_t max_clusters, int64_t n, const int32_t* x,
                                          const int32_t* y, const int8_t* c, const float* r, float threshold,
                                          float* eigens, int32_t* size)
{
   if ( !eigens || !size ) return rmt_fail(KINC_SIM_EINVAL, "invalid arguments");
   RmtDevice d;
   int rc = device_setup(d, genes, max_clusters, n, x, y, c, r);
   if ( rc ) return rc;
   std::vector<float> e;
   int32_t m = 0;
   if ( (rc = device_eigenvalues(d, threshold, e, m)) ) return rc;
   std::copy(e.begin(), e.end(), eigens);
   *size = m;
   return KINC_SIM_OK;
}

extern "C" int kinc_rmt_run_items(int32_t genes, int32_t max_clusters, int64_t n, const int32_t* x, const int32_t* y,
                                  const int8_t* c, const float* r, const kinc_rmt_params* p, const char* log_path,
                                  float* out_threshold, float* steps_out, int32_t steps_cap, int32_t* steps)
{
   int rc = check_params(p);
   if ( rc ) return rc;
   if ( !out_threshold ) return rmt_fail(KINC_SIM_EINVAL, "out_threshold must not be NULL");
   RmtDevice d;
   if ( (rc = device_setup(d, genes, max_clusters, n, x, y, c, r)) ) return rc;
   FILE* log = nullptr;
   if ( log_path && !(log = fopen(log_path, "wb")) ) return rmt_fail(KINC_SIM_EINVAL, "cannot open %s", log_path);

   /* RMT::process: thresholds downwards until a large chi-square follows a small one */
   float finalThreshold = 0.0f;
   float finalChi = std::numeric_limits<float>::infinity();
   float maxChi = -std::numeric_limits<float>::infinity();
   float threshold = p->threshold_start;
   int32_t nsteps = 0;
   std::vector<float> eig;
   while ( maxChi < p->chi_square_threshold2 )
   {
      int32_t m = 0;
      if ( (rc = device_eigenvalues(d, threshold, eig, m)) ) break;
      float chi = -1.0f;
      if ( m > 0 && (rc = chi_square(eig.data(), m, *p, chi)) ) break;
      if ( chi != -1.0f )
      {
         if ( chi < p->chi_square_threshold1 )
         {
            finalChi = chi;
            finalThreshold = threshold;
         }
         if ( finalChi < p->chi_square_threshold1 && chi > finalChi ) maxChi = chi;
      }
      if ( log ) fprintf(log, "%.6g\t%d\t%.6g\n", (double)threshold, m, (double)chi);
      if ( steps_out && nsteps < steps_cap )
      {
         steps_out[3 * nsteps] = threshold;
         steps_out[3 * nsteps + 1] = (float)m;
         steps_out[3 * nsteps + 2] = chi;
      }
      ++nsteps;
      threshold -= p->threshold_step;
      if ( threshold < p->threshold_stop )
      {
         rc = rmt_fail(KINC_RMT_ENOTHRESHOLD, "Could not find non-random threshold above stopping threshold.");
         break;
      }
   }
   if ( log )
   {
      if ( rc == KINC_SIM_OK ) fprintf(log, "%.6g\n", (double)finalThreshold);
      fclose(log);
   }
   if ( steps ) *steps = nsteps;
   *out_threshold = finalThreshold;
   return rc;
}

extern "C" int kinc_rmt_run(const char* cmx_path, int32_t little_endian, const kinc_rmt_params* p, const char* log_path,
                            float* out_threshold)
{
   kinc_pm* m = nullptr;
   int32_t G = 0, K = 0, nc = 0;
   int64_t pairs = 0, n = 0;
   int rc = kinc_pm_open(cmx_path, KINC_PM_CMX, little_endian, &m, &G, &K, &nc, &pairs, &n);
   if ( rc ) return rmt_fail(rc, "%s", kinc_pm_last_error());
   std::vector<int32_t> x((size_t)std::max<int64_t>(n, 1)), y((size_t)std::max<int64_t>(n, 1));
   std::vector<int8_t> c((size_t)std::max<int64_t>(n, 1));
   std::vector<float> all((size_t)std::max<int64_t>(n, 1) * std::max(nc, 1)), r((size_t)std::max<int64_t>(n, 1));
   rc = n > 0 ? kinc_pm_read_items(m, 0, n, x.data(), y.data(), c.data(), all.data()) : KINC_SIM_OK;
   kinc_pm_close(m);
   if ( rc ) return rmt_fail(rc, "%s", kinc_pm_last_error());
   for ( int64_t i = 0; i < n; ++i ) r[(size_t)i] = all[(size_t)i * nc];   /* the first correlation */
   return kinc_rmt_run_items(G, K, n, x.data(), y.data(), c.data(), r.data(), p, log_path, out_threshold, nullptr, 0,
                             nullptr);
}
