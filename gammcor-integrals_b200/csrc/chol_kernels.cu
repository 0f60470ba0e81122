// chol_kernels.cu -- device kernels of the two-step Cholesky driver:
// candidate compression, the batch pivot search, the downdate of the
// diagonal and the reshaping kernels of the AO->MO transformation.
#include "gci_common.h"
#include "gci_runtime.h"
#include <algorithm>
#include <cfloat>

namespace gci {

// Max of D over each shell pair's orbital-pair segment (DefineCandidates /
// DefineBatch, TwoStepCholesky_Step1.f90:547-552,600-605).
__global__ void k_segmax(const double* __restrict__ D, const int64_t* __restrict__ loc,
                         const int* __restrict__ dim, int64_t n, double* __restrict__ out)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double* d = D + loc[i];
        double m = -DBL_MAX;
        for (int k = 0; k < dim[i]; ++k) m = fmax(m, d[k]);
        out[i] = m;
    }
}

// new[i + ldn*j] = old[src[i] + ldo*j], i < nrows, j < ncols (chol2_Compress).
__global__ void k_gather_rows(const double* __restrict__ src_mat, int64_t ld_src, const int64_t* __restrict__ src,
                              int64_t nrows, int64_t ncols, double* __restrict__ dst, int64_t ld_dst)
{
    const int64_t total = nrows * ncols;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t j = t / nrows, i = t - j * nrows;
        dst[i + ld_dst * j] = src_mat[src[i] + ld_src * j];
    }
}

// dst[r + ld_dst*j] = src[r + ld_src*cols[j]] (pivot columns of M)
__global__ void k_gather_cols(const double* __restrict__ src, int64_t ld_src, const int* __restrict__ cols,
                              int64_t nrows, int64_t ncols, double* __restrict__ dst, int64_t ld_dst)
{
    const int64_t total = nrows * ncols;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t j = t / nrows, r = t - j * nrows;
        dst[r + ld_dst * j] = src[r + ld_src * cols[j]];
    }
}

__device__ __forceinline__ bool better(double v, int i, double bv, int bi)
{
    return v > bv || (v == bv && i < bi);
}

// Micro-iterations of one macro iteration (chol2_Pivots, Step1.f90:1025-1064)
// restricted to the batch: the pivot choice depends only on the batch rows
// of M and of the new vectors, so the sequential part runs on the nb x nb
// block Mbb; the vectors over all candidates follow afterwards as one
// triangular solve.  Lb(:, j) = (Mbb(:, piv_j) - Lb Lb(piv_j, :)^T) / sqrt(Dmax_j).
//
// Every pivot needs all previous vectors of its row and of every other row, so
// the search is bound by how fast Lb can be re-read, pivot after pivot.  One
// cluster of kPivCtas blocks holds it: each keeps its rows of Lb (the first jcap
// vectors) and of the diagonal in shared memory, four lanes a row.  Per pivot
// one exchange of the blocks' maxima through distributed shared memory (with
// the reference's tie rule: strict '>' in increasing index order, chol2_BatchMax,
// TwoStepCholesky_Step1.f90:720-727) and one read of the pivot's row from its owner.
// About 3.5 us a pivot, most of it the two exchanges; one block that reads Lb back from
// L2 took 9 ms for a batch of 1000 rows (pivot phase of 10 atoms, 140 AOs: 20.4 -> 9.0 ms;
// of 12 atoms, 360 AOs with f shells: 115 -> 53 ms).
constexpr int kPivCtas = 8, kPivThreads = 512, kPivSub = 4, kPivRowsPerPass = kPivThreads / kPivSub;

__device__ __forceinline__ void cluster_barrier()
{
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// address of this block's shared variable `p` in block `rank` of the cluster
__device__ __forceinline__ uint32_t cluster_addr(const void* p, int rank)
{
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_store(uint32_t a, double v)
{
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void cluster_store(uint32_t a, int v)
{
    asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ double cluster_load(uint32_t a)
{
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
    return v;
}

__global__ void __cluster_dims__(kPivCtas, 1, 1) __launch_bounds__(kPivThreads, 1)
k_pivot_batch(const double* __restrict__ Mbb, int nb, const double* __restrict__ Db, double* __restrict__ Lb,
              int* __restrict__ piv, double* __restrict__ pdmax, int* __restrict__ npiv_out, int64_t nchol0,
              int64_t maxnchol, double dmin, int rpc, int pitch, int jcap)
{
    // rows [row0, row0 + nr) of the batch: rpc a block
    extern __shared__ __align__(16) double sh[];
    double* prow = sh;                          // nb: the pivot's row of the vectors so far
    double* Ds = prow + nb;                     // rpc: residual diagonal of the block's rows
    double* Ls = Ds + rpc;                      // jcap x pitch: vectors of the block's rows
    __shared__ double x_v[2][kPivCtas];         // the blocks' maxima, alternating between pivots
    __shared__ int x_i[2][kPivCtas];
    const int rank = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row0 = rank * rpc, nr = min(rpc, nb - row0);   // nr <= 0: no rows
    for (int r = tid; r < nr; r += kPivThreads) Ds[r] = Db[row0 + r];
    // a warp takes 8 rows of 4 lanes; the lanes of a row take every fourth vector
    const int sub = lane >> 3, rl = warp * 8 + (lane & 7);

    // maximum over all rows of the batch and its first index, the same in every thread
    auto argmax = [&](int par, double& bv, int& bi) {
        __syncthreads();
        if (warp == 0) {
            double v = -DBL_MAX;
            int i = 0x7fffffff;
            for (int r = lane; r < nr; r += 32)
                if (better(Ds[r], row0 + r, v, i)) { v = Ds[r]; i = row0 + r; }
            for (int off = 16; off > 0; off >>= 1) {
                const double ov = __shfl_xor_sync(0xffffffffu, v, off);
                const int oi = __shfl_xor_sync(0xffffffffu, i, off);
                if (better(ov, oi, v, i)) { v = ov; i = oi; }
            }
            if (lane < kPivCtas) {
                cluster_store(cluster_addr(&x_v[par][rank], lane), v);
                cluster_store(cluster_addr(&x_i[par][rank], lane), i);
            }
            __syncwarp();
        }
        cluster_barrier();   // the maxima are exchanged, and every block's vectors so far are complete
        bv = -DBL_MAX;
        bi = 0x7fffffff;
#pragma unroll
        for (int c = 0; c < kPivCtas; ++c)
            if (better(x_v[par][c], x_i[par][c], bv, bi)) { bv = x_v[par][c]; bi = x_i[par][c]; }
    };

    double maxv;
    int maxi;
    cluster_barrier();   // every block of the cluster runs before its shared memory is written
    argmax(0, maxv, maxi);
    int j = 0;
    bool go = (nchol0 < maxnchol) && maxi < nb;
    while (go) {
        if (rank == 0 && tid == 0) { piv[j] = maxi; pdmax[j] = maxv; }
        const int owner = maxi / rpc, orow = maxi - owner * rpc;
        const int js = min(j, jcap);
        for (int i = tid; i < js; i += kPivThreads) prow[i] = cluster_load(cluster_addr(Ls + (size_t)i * pitch + orow, owner));
        for (int i = js + tid; i < j; i += kPivThreads) prow[i] = __ldcg(Lb + maxi + (int64_t)nb * i);
        __syncthreads();
        const double sq = sqrt(maxv);
        for (int r = rl; r < rpc; r += kPivRowsPerPass) {   // uniform within a warp up to the row bound
            const bool on = r < nr;
            double s0 = 0.0, s1 = 0.0;
            if (on) {
                if (sub == 0) s0 = Mbb[row0 + r + (int64_t)nb * maxi];
                int i = sub;
                for (; i + kPivSub < js; i += 2 * kPivSub) {
                    s0 = fma(-Ls[(size_t)i * pitch + r], prow[i], s0);
                    s1 = fma(-Ls[(size_t)(i + kPivSub) * pitch + r], prow[i + kPivSub], s1);
                }
                for (; i < js; i += kPivSub) s0 = fma(-Ls[(size_t)i * pitch + r], prow[i], s0);
                for (i = js + sub; i < j; i += kPivSub) s1 = fma(-__ldcg(Lb + row0 + r + (int64_t)nb * i), prow[i], s1);
            }
            double s = s0 + s1;
            s += __shfl_xor_sync(0xffffffffu, s, 8);
            s += __shfl_xor_sync(0xffffffffu, s, 16);
            if (on && sub == 0) {
                const double l = s / sq;
                if (j < jcap) Ls[(size_t)j * pitch + r] = l;
                __stcg(Lb + row0 + r + (int64_t)nb * j, l);
                Ds[r] -= l * l;
            }
        }
        ++j;
        argmax(j & 1, maxv, maxi);
        if (maxv <= dmin) go = false;
        if (j == nb || nchol0 + j == maxnchol) go = false;
    }
    if (rank == 0 && tid == 0) *npiv_out = j;
}

// Lp(j, i) = Lb(piv[j], i): the pivot rows of the new vectors (lower triangular)
__global__ void k_gather_pivrows(const double* __restrict__ Lb, int nb, const int* __restrict__ piv, int npiv,
                                 double* __restrict__ Lp)
{
    const int64_t total = (int64_t)npiv * npiv;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(t / npiv), jr = (int)(t - (int64_t)i * npiv);
        Lp[jr + (int64_t)npiv * i] = (i <= jr) ? Lb[piv[jr] + (int64_t)nb * i] : 0.0;
    }
}

// Inverse of a lower-triangular n x n matrix, one block per column
// (forward substitution with a block reduction per row).
__global__ void k_tri_inv_lower(const double* __restrict__ L, int n, double* __restrict__ X)
{
    __shared__ double red[32];
    __shared__ double xcol_s;
    for (int c = blockIdx.x; c < n; c += gridDim.x) {
        double* xc = X + (int64_t)n * c;
        for (int i = threadIdx.x; i < c; i += blockDim.x) xc[i] = 0.0;
        if (threadIdx.x == 0) xc[c] = 1.0 / L[c + (int64_t)n * c];
        __syncthreads();
        for (int i = c + 1; i < n; ++i) {
            double s = 0.0;
            for (int k = c + threadIdx.x; k < i; k += blockDim.x) s += L[i + (int64_t)n * k] * xc[k];
            for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
            if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
            __syncthreads();
            if (threadIdx.x == 0) {
                double t = 0.0;
                for (int w = 0; w < (int)((blockDim.x + 31) >> 5); ++w) t += red[w];
                xcol_s = -t / L[i + (int64_t)n * i];
                xc[i] = xcol_s;
            }
            __syncthreads();
        }
    }
}

// D[r] -= sum_j L[r + ld*j]^2  (D(:) = D(:) - Lpqj(:,j)**2, Step1.f90:1046)
__global__ void k_downdate(double* __restrict__ D, const double* __restrict__ L, int64_t ld, int64_t n, int ncols)
{
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
        double d = D[r];
        for (int j = 0; j < ncols; ++j) {
            const double l = L[r + ld * j];
            d -= l * l;
        }
        D[r] = d;
    }
}

__global__ void k_max(const double* __restrict__ v, int64_t n, double* __restrict__ out)
{
    __shared__ double red[32];
    double m = -DBL_MAX;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) m = fmax(m, v[i]);
    for (int off = 16; off > 0; off >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, off));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = -DBL_MAX;
        for (int w = 0; w < (int)((blockDim.x + 31) >> 5); ++w) t = fmax(t, red[w]);
        *out = t;
    }
}

__global__ void k_zero_upper(double* __restrict__ A, int64_t n)
{
    const int64_t total = n * n;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t j = t / n, i = t - j * n;
        if (i < j) A[t] = 0.0;
    }
}

// A(i, j) = A(j, i) where rank[i] > rank[j], through 32 x 32 tiles in shared memory so that both
// sides are read and written in runs (bound by HBM: half of A read, half written).
__global__ void __launch_bounds__(256) k_mirror(double* __restrict__ A, int64_t ld, int64_t n,
                                                const int* __restrict__ rank)
{
    __shared__ double t[32][33];
    const int64_t i0 = (int64_t)blockIdx.x * 32, j0 = (int64_t)blockIdx.y * 32;   // destination tile A(i0.., j0..)
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
    for (int k = y; k < 32; k += 8)
        if (j0 + x < n && i0 + k < n) t[k][x] = A[(j0 + x) + ld * (i0 + k)];
    __syncthreads();
    for (int k = y; k < 32; k += 8) {
        const int64_t i = i0 + x, j = j0 + k;
        if (i < n && j < n && __ldg(rank + i) > __ldg(rank + j)) A[i + ld * j] = t[x][k];
    }
}

// Unpack Rkpq(k, pq) (k in [k0, k0+kc)) into the dense symmetric AO-pair
// layout U[p][q][k - k0] (both triangles) for the AO->MO GEMMs.
// One entry per stored orbital pair: pq_ao[2*i] = p, pq_ao[2*i+1] = q, and
// pq_col[i] = column of the pair in the (NVecs x MaxSubsetDim x NSubsets) array.
__global__ void k_unpack_rkpq(const double* __restrict__ R, int64_t nvecs, const int64_t* __restrict__ pq_col,
                              const int* __restrict__ pq_ao, int64_t npq, int64_t k0, int64_t kc, int64_t nao,
                              double* __restrict__ U)
{
    const int64_t total = npq * kc;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = t / kc, k = t - i * kc;
        const double v = R[(k0 + k) + nvecs * pq_col[i]];
        const int64_t p = pq_ao[2 * i], q = pq_ao[2 * i + 1];
        U[(p * nao + q) * kc + k] = v;
        if (p != q) U[(q * nao + p) * kc + k] = v;
    }
}

static inline unsigned grid_for(int64_t n, int threads, int64_t cap = 148LL * 32)
{
    int64_t b = (n + threads - 1) / threads;
    if (b < 1) b = 1;
    if (b > cap) b = cap;
    return (unsigned)b;
}

cudaError_t launch_segmax(const double* D, const int64_t* loc, const int* dim, int64_t n, double* out, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    k_segmax<<<grid_for(n, 256), 256, 0, s>>>(D, loc, dim, n, out);
    count_launch();
    return cudaGetLastError();
}
cudaError_t launch_gather_rows(const double* src, int64_t lds, const int64_t* idx, int64_t nrows, int64_t ncols,
                               double* dst, int64_t ldd, cudaStream_t s)
{
    if (nrows <= 0 || ncols <= 0) return cudaSuccess;
    k_gather_rows<<<grid_for(nrows * ncols, 256), 256, 0, s>>>(src, lds, idx, nrows, ncols, dst, ldd);
    count_launch();
    return cudaGetLastError();
}
cudaError_t launch_gather_cols(const double* src, int64_t lds, const int* cols, int64_t nrows, int64_t ncols,
                               double* dst, int64_t ldd, cudaStream_t s)
{
    if (nrows <= 0 || ncols <= 0) return cudaSuccess;
    k_gather_cols<<<grid_for(nrows * ncols, 256), 256, 0, s>>>(src, lds, cols, nrows, ncols, dst, ldd);
    count_launch();
    return cudaGetLastError();
}
cudaError_t launch_pivot_batch(const double* Mbb, int nb, double* Db, double* Lb, int* piv, double* pdmax,
                               int* npiv, int64_t nchol0, int64_t maxnchol, double dmin, cudaStream_t s)
{
    // rows a block (a multiple of a warp's 8); the pitch 8 mod 16 keeps the four lanes of a row
    // and the eight rows of a warp in different banks; as many vectors as fit 200 KB
    const int rpc = std::max(8, ((nb + kPivCtas - 1) / kPivCtas + 7) / 8 * 8);
    const int pitch = (rpc + 15) / 16 * 16 + 8;
    const int64_t room = (int64_t)(200 * 1024) / 8 - nb - rpc;
    const int jcap = room > 0 ? (int)std::min<int64_t>(nb, room / pitch) : 0;
    const size_t smem = sizeof(double) * ((size_t)nb + rpc + (size_t)jcap * pitch);
    // the same value from every caller: workers of a batch launch at the same time
    cudaError_t e = cudaFuncSetAttribute(k_pivot_batch, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
    if (e != cudaSuccess) return e;
    k_pivot_batch<<<kPivCtas, kPivThreads, smem, s>>>(Mbb, nb, Db, Lb, piv, pdmax, npiv, nchol0, maxnchol, dmin, rpc,
                                                      pitch, jcap);
    count_launch();
    return cudaGetLastError();
}
cudaError_t launch_gather_pivrows(const double* Lb, int nb, const int* piv, int npiv, double* Lp, cudaStream_t s)
{
    if (npiv <= 0) return cudaSuccess;
    k_gather_pivrows<<<grid_for((int64_t)npiv * npiv, 256), 256, 0, s>>>(Lb, nb, piv, npiv, Lp);
    count_launch();
    return cudaGetLastError();
}
cudaError_t launch_tri_inv_lower(const double* L, int n, double* X, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    k_tri_inv_lower<<<n < 148 * 8 ? n : 148 * 8, 128, 0, s>>>(L, n, X);
    count_launch();
    return cudaGetLastError();
}
cudaError_t launch_downdate(double* D, const double* L, int64_t ld, int64_t n, int ncols, cudaStream_t s)
{
    if (n <= 0 || ncols <= 0) return cudaSuccess;
    k_downdate<<<grid_for(n, 256), 256, 0, s>>>(D, L, ld, n, ncols);
    count_launch();
    return cudaGetLastError();
}
cudaError_t launch_max(const double* v, int64_t n, double* out, cudaStream_t s)
{
    k_max<<<1, 1024, 0, s>>>(v, n, out);
    count_launch();
    return cudaGetLastError();
}
cudaError_t launch_mirror(double* A, int64_t ld, int64_t n, const int* rank, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    const unsigned g = (unsigned)((n + 31) / 32);
    if (g > 65535) return cudaErrorInvalidValue;
    k_mirror<<<dim3(g, g), 256, 0, s>>>(A, ld, n, rank);
    count_launch();
    return cudaGetLastError();
}
cudaError_t launch_zero_upper(double* A, int64_t n, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    k_zero_upper<<<grid_for(n * n, 256), 256, 0, s>>>(A, n);
    count_launch();
    return cudaGetLastError();
}
cudaError_t launch_unpack_rkpq(const double* R, int64_t nvecs, const int64_t* pq_col, const int* pq_ao, int64_t npq,
                               int64_t k0, int64_t kc, int64_t nao, double* U, cudaStream_t s)
{
    if (npq <= 0 || kc <= 0) return cudaSuccess;
    k_unpack_rkpq<<<grid_for(npq * kc, 256), 256, 0, s>>>(R, nvecs, pq_col, pq_ao, npq, k0, kc, nao, U);
    count_launch();
    return cudaGetLastError();
}

} // namespace gci
