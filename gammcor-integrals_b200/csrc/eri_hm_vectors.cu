// eri_hm_vectors.cu -- the pair Hermite vectors of the Hermite-matrix ERI
// kernels (eri_hermite.cuh) and the launch table of those kernels.
//
// A vector element is the Hermite coefficient of one (spherical, normalised)
// function pair of a primitive pair,
//     K c c sum_{a in A, b in B} T_A(f_a, a) T_B(f_b, b) Ex^{ab}_t Ey^{ab}_u Ez^{ab}_v,
// the normalisation and solid-harmonic transforms of the reference
// (auto2e_SpherTransf.f90, auto2e_Normalize_*, sphergto.f90:184-211)
// applied to the two-centre Hermite coefficients of the primitive-pair
// record (k_pair_records).  Elements are written directly in the fragment
// order the DMMA products read.
#include "eri_hermite.cuh"
#include "gci_runtime.h"
#include <mutex>

namespace gci {

// Index tables of a pair in shared memory: the powers of the Cartesian
// components and of the Hermite indices, and the nonzero entries of the two
// shells' transforms (one to three of the ncart(l) for most solid harmonics).
// Elements are cheap sums over these lists, bound by the latency of their table
// loads; decoding the indices and scanning the dense transforms for every
// element cost several times the arithmetic (ERI matrix of 60 AOs with f shells
// 63 -> 40 ms, the AO->MO transform at 210 AOs 237 -> 211 ms).
struct HmPairTab {
    int herm[herm_n(kMaxPairL)];              // t | u << 8 | v << 16
    int nz[2][2 * kMaxL + 1];                 // nonzero entries of each function
    int pw[2][2 * kMaxL + 1][ncart(kMaxL)];   // their powers x | y << 8 | z << 16
    double w[2][2 * kMaxL + 1][ncart(kMaxL)]; // and weights, in the order of the components
};

// Fills the table for the pair d (all threads of the block; synchronises).
__device__ static void hm_pair_tab(HmPairTab& T, const ShellPairDev& d, const double* __restrict__ tmat,
                                   const int* __restrict__ toff, const int* __restrict__ nfunc)
{
    __syncthreads();   // the previous pair's readers are done
    const int H = herm_n(d.l1 + d.l2);
    for (int h = threadIdx.x; h < H; h += blockDim.x) T.herm[h] = herm_t(h) | (herm_u(h) << 8) | (herm_v(h) << 16);
    if (threadIdx.x < 2 * (2 * kMaxL + 1)) {
        const int which = threadIdx.x / (2 * kMaxL + 1), f = threadIdx.x % (2 * kMaxL + 1);
        const int s = which ? d.s2 : d.s1, l = which ? d.l2 : d.l1, nc = ncart(l);
        int n = 0;
        if (f < __ldg(nfunc + s)) {
            const double* __restrict__ t = tmat + __ldg(toff + s) + f * nc;
            for (int c = 0; c < nc; ++c) {
                const double w = __ldg(t + c);
                if (w == 0.0) continue;
                const int g = cart_off(l) + c;
                T.pw[which][f][n] = cart_x(g) | (cart_y(g) << 8) | (cart_z(g) << 16);
                T.w[which][f][n] = w;
                ++n;
            }
        }
        T.nz[which][f] = n;
    }
    __syncthreads();
}

// Coefficient of Hermite index (t,u,v) (packed) of the function pair (f1, f2) of the
// canonical shells (s1, s2) of a pair in primitive-pair record `rec`.
__device__ static double hm_element(const HmPairTab& T, const ShellPairDev& d, const double* __restrict__ rec, int f1,
                                    int f2, int tuv)
{
    const int la = d.l1, ne = e2_size(la, d.l2);
    const int t = tuv & 255, u = (tuv >> 8) & 255, v = tuv >> 16;
    const double* __restrict__ Ex = rec + 8 + t;
    const double* __restrict__ Ey = rec + 8 + ne + u;
    const double* __restrict__ Ez = rec + 8 + 2 * ne + v;
    double sum = 0.0;
    for (int c1 = 0; c1 < T.nz[0][f1]; ++c1) {
        const double w1 = T.w[0][f1][c1];
        const int p1 = T.pw[0][f1][c1], x1 = p1 & 255, y1 = (p1 >> 8) & 255, z1 = p1 >> 16;
        for (int c2 = 0; c2 < T.nz[1][f2]; ++c2) {
            const double w2 = T.w[1][f2][c2];
            const int p2 = T.pw[1][f2][c2], x2 = p2 & 255, y2 = (p2 >> 8) & 255, z2 = p2 >> 16;
            if (t > x1 + x2 || u > y1 + y2 || v > z1 + z2) continue;
            sum += w1 * w2 * __ldg(Ex + e2_off(la, x1, x2)) * __ldg(Ey + e2_off(la, y1, y2)) *
                   __ldg(Ez + e2_off(la, z1, z2));
        }
    }
    return sum * __ldg(rec + 4);
}

// Stored-orientation function code f = f_first + N_first f_second -> canonical (f1, f2).
__device__ __forceinline__ void hm_canon(const ShellPairDev& d, const int* __restrict__ nfunc, int f, int& f1, int& f2)
{
    const int first = d.swap ? d.s2 : d.s1;
    const int nfirst = __ldg(nfunc + first);
    const int fa = f % nfirst, fb = f / nfirst;
    f1 = d.swap ? fb : fa;
    f2 = d.swap ? fa : fb;
}

// Row vectors of the listed pairs: per block of primitive pairs [MTO][2 MT][32], element
// (m, 2 j + e, l) = Er(r = 8 m + l/4, (i,h) = 8 j + 2 (l%4) + e) -- the k order in which the
// accumulators of the first product are the B fragments of the second; one block per pair.
__global__ void k_hm_rowvec(const int* __restrict__ ids, int nids, const ShellPairDev* __restrict__ pairs,
                            const double* __restrict__ pp, const int64_t* __restrict__ off,
                            const double* __restrict__ tmat, const int* __restrict__ toff,
                            const int* __restrict__ nfunc, double* __restrict__ vec)
{
    __shared__ HmPairTab T;
    for (int q = blockIdx.x; q < nids; q += gridDim.x) {
        const int id = ids[q];
        const ShellPairDev d = pairs[id];
        const int L = d.l1 + d.l2;
        const int H = herm_n(L), MT2 = 2 * hm_mt(L), stride = hm_row_stride(L), IB = hm_ib(L);
        const int nR = __ldg(nfunc + d.s1) * __ldg(nfunc + d.s2);
        const int rs = pp_record(d.l1, d.l2);
        hm_pair_tab(T, d, tmat, toff, nfunc);
        double* __restrict__ out = vec + off[id];
        const int64_t n = (int64_t)hm_row_blocks(L, d.npp) * stride;
        for (int64_t e = threadIdx.x; e < n; e += blockDim.x) {
            const int ib = (int)(e / stride);
            const int w = (int)(e - (int64_t)ib * stride);
            const int l = w & 31, f = w >> 5;
            const int m = f / MT2, ks = f - m * MT2;
            const int r = 8 * m + (l >> 2), rho = 8 * (ks >> 1) + 2 * (l & 3) + (ks & 1);
            const int il = rho / H, h = rho - il * H, i = ib * IB + il;
            double val = 0.0;
            if (r < nR && il < IB && i < d.npp) {
                int f1, f2;
                hm_canon(d, nfunc, r, f1, f2);
                val = hm_element(T, d, pp + d.rec_off + (size_t)i * rs, f1, f2, T.herm[h]);
            }
            out[e] = val;
        }
    }
}

// Column vectors of the chunks: per group of primitive pairs [KT][NT][32], element
// (ks, n, l) = (-1)^|g| Ec((k,g) = 4 ks + l%4, J = 8 n + l/4); one block per chunk.
__global__ void k_hm_colvec(const HmChunk* __restrict__ chunks, int nchunks, const ShellPairDev* __restrict__ pairs,
                            const double* __restrict__ pp, const int* __restrict__ colfun,
                            const double* __restrict__ tmat, const int* __restrict__ toff,
                            const int* __restrict__ nfunc, double* __restrict__ vec)
{
    __shared__ HmPairTab T;
    for (int q = blockIdx.x; q < nchunks; q += gridDim.x) {
        const HmChunk ch = chunks[q];
        const ShellPairDev d = pairs[ch.pair];
        const int L = d.l1 + d.l2;
        const int H = herm_n(L), stride = hm_col_stride(L, ch.nt), KP = hm_kp(L);
        const int rs = pp_record(d.l1, d.l2);
        hm_pair_tab(T, d, tmat, toff, nfunc);
        double* __restrict__ out = vec + ch.vec_off;
        const int64_t n = (int64_t)hm_col_groups(L, d.npp) * stride;
        for (int64_t e = threadIdx.x; e < n; e += blockDim.x) {
            const int kg = (int)(e / stride);
            const int w = (int)(e - (int64_t)kg * stride);
            const int l = w & 31, f = w >> 5;
            const int ks = f / ch.nt, nn = f - ks * ch.nt;
            const int kap = 4 * ks + (l & 3), J = 8 * nn + (l >> 2);
            const int kl = kap / H, g = kap - kl * H, k = kg * KP + kl;
            double val = 0.0;
            if (kl < KP && k < d.npp && J < ch.ncol) {
                int f1, f2;
                hm_canon(d, nfunc, colfun[ch.col_off + J], f1, f2);
                const int tuv = T.herm[g];
                val = hm_element(T, d, pp + d.rec_off + (size_t)k * rs, f1, f2, tuv);
                if ((tuv ^ (tuv >> 8) ^ (tuv >> 16)) & 1) val = -val;
            }
            out[e] = val;
        }
    }
}

cudaError_t hm_rowvec_launch(const int* ids, int nids, const ShellPairDev* pairs, const double* pp,
                             const int64_t* off, const double* tmat, const int* toff, const int* nfunc, double* vec,
                             cudaStream_t st)
{
    if (nids <= 0) return cudaSuccess;
    const int blocks = nids < 148 * 32 ? nids : 148 * 32;
    k_hm_rowvec<<<blocks, 256, 0, st>>>(ids, nids, pairs, pp, off, tmat, toff, nfunc, vec);
    count_launch();
    return cudaGetLastError();
}

cudaError_t hm_colvec_launch(const HmChunk* chunks, int nchunks, const ShellPairDev* pairs, const double* pp,
                             const int* colfun, const double* tmat, const int* toff, const int* nfunc, double* vec,
                             cudaStream_t st)
{
    if (nchunks <= 0) return cudaSuccess;
    const int blocks = nchunks < 148 * 32 ? nchunks : 148 * 32;
    k_hm_colvec<<<blocks, 256, 0, st>>>(chunks, nchunks, pairs, pp, colfun, tmat, toff, nfunc, vec);
    count_launch();
    return cudaGetLastError();
}

static HmLaunch g_hm[kMaxPairL + 1][kMaxPairL + 1][kHmMaxNT];

static const HmLaunch* hm_class(int L1, int L2, int nt)
{
    static std::once_flag once;
    std::call_once(once, [] {
        register_hm_0(g_hm);
        register_hm_1(g_hm);
        register_hm_2(g_hm);
        register_hm_3(g_hm);
        register_hm_4(g_hm);
        register_hm_5(g_hm);
        register_hm_6(g_hm);
    });
    if (L1 < 0 || L2 < 0 || L1 > kMaxPairL || L2 > kMaxPairL || nt < 1 || nt > hm_max_nt(L1)) return nullptr;
    const HmLaunch* h = &g_hm[L1][L2][nt - 1];
    return h->launch ? h : nullptr;
}

int hm_split(int L1, int L2, int nt, int64_t ntasks, int nib, int nkg, int64_t& doubles)
{
    const HmLaunch* h = hm_class(L1, L2, nt);
    doubles = 0;
    if (!h || ntasks <= 0) return 1;
    const int64_t want = h->resident();
    if (ntasks >= want) return 1;
    // a part's tensor-core products: below about 4000 (64k cycles of one SM quarter) its own start
    // and the exchange of its block through L2 are no longer small beside them.  Measured, step-1
    // integrals: 60 AOs with f shells 95 ms in whole tasks, 37 with this rule; parts down to one
    // block in every launch below three rounds of the resident warps took 140 AOs from 11.9 to
    // 23.4 ms, parts for four rounds (of at least 8000 products) 360 AOs from 600 to 717 ms.
    constexpr int64_t kMinProducts = 4000;
    const int64_t products = (int64_t)nib * nkg * hm_kt(L2) * hm_mt(L1) * nt;
    int64_t split = std::min<int64_t>((want + ntasks - 1) / ntasks, nib);
    split = std::min<int64_t>(split, products / kMinProducts);
    if (split <= 1) return 1;
    doubles = ntasks * split * h->block;
    return (int)split;
}

cudaError_t hm_launch(int L1, int L2, int nt, const HmArgs& a, cudaStream_t st)
{
    const HmLaunch* h = hm_class(L1, L2, nt);
    if (!h) return cudaErrorInvalidValue;
    const cudaError_t e = h->launch(a, st);
    count_launch();
    return e;
}

} // namespace gci
