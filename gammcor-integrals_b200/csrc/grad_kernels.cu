// grad_kernels.cu -- density-contracted Hermite vectors, the dot products that
// give the Coulomb energy and its nuclear gradient, the Coulomb matrix, and
// the dispatch table of the potential kernels (grad_engine.cuh,
// instantiated in grad_pot_*.cu).
#include "grad_engine.cuh"
#include "gci_runtime.h"
#include <mutex>

namespace gci {

// E^{ij}_t of one axis for i <= la + 1, j <= lb + 1 (t <= i + j; zero beyond):
// the two-centre McMurchie-Davidson recursion in P-A and P-B with
// E^{00}_0 = 1 (the Gaussian product factor is applied separately).
struct GradE {
    static constexpr int NI = kMaxL + 2, NT = 2 * kMaxL + 3;
    double e[NI][NI][NT];
};

// Fills a table that is zero on entry.
__device__ static void grad_etab(GradE& E, int la, int lb, double PA, double PB, double h)
{
    E.e[0][0][0] = 1.0;
    for (int i = 0; i <= la; ++i)
        for (int t = 0; t <= i + 1; ++t) {
            double v = PA * E.e[i][0][t];
            if (t >= 1) v += h * E.e[i][0][t - 1];
            if (t + 1 <= i) v += (double)(t + 1) * E.e[i][0][t + 1];
            E.e[i + 1][0][t] = v;
        }
    for (int j = 0; j <= lb; ++j)
        for (int i = 0; i <= la + 1; ++i)
            for (int t = 0; t <= i + j + 1; ++t) {
                double v = PB * E.e[i][j][t];
                if (t >= 1) v += h * E.e[i][j][t - 1];
                if (t + 1 <= i + j) v += (double)(t + 1) * E.e[i][j][t + 1];
                E.e[i][j + 1][t] = v;
            }
}

// One block per shell pair: the Cartesian density block Ds (symmetrised,
// times w_AB, with the norms and spherical transforms of both shells) in
// shared memory, then one warp per kept primitive pair writes its seven
// Hermite vectors (h, gA, gB; grad_hb(L) entries each), its geometry and,
// transposed and signed, its ket vector: three lanes fill the axes' tables in
// shared memory, then each lane sums whole entries over the Cartesian pairs in
// registers.  (One thread per primitive pair, with its tables in local memory
// and its entries accumulated in global memory, is a chain of thousands of
// dependent accesses.)  80 us on 42 AOs, latency of the tables' recursion.
constexpr int kGradVecWarps = 2;
__global__ void k_grad_pair_vectors(const ShellPairDev* __restrict__ pairs, int npairs,
                                    const int64_t* __restrict__ gbase, const int* __restrict__ level_beg,
                                    const int* __restrict__ level_n, const int64_t* __restrict__ vec_off,
                                    const int64_t* __restrict__ hk_off, const double* __restrict__ xyz,
                                    const int* __restrict__ poff, const double* __restrict__ exps,
                                    const double* __restrict__ coefs, const int* __restrict__ plist,
                                    const double* __restrict__ tmat, const int* __restrict__ toff,
                                    const int* __restrict__ nfunc, const int* __restrict__ loc,
                                    const double* __restrict__ D, int64_t ldd, double* __restrict__ mP,
                                    double* __restrict__ mX, double* __restrict__ mY, double* __restrict__ mZ,
                                    double* __restrict__ vecs, double* __restrict__ hk, int* __restrict__ ppair)
{
    __shared__ double Dc[ncart(kMaxL) * ncart(kMaxL)];
    __shared__ int cart[2][ncart(kMaxL)];            // x | y << 8 | z << 16 of the components of both shells
    __shared__ int herm[grad_hb(2 * kMaxL)];         // t | u << 8 | v << 16
    __shared__ GradE tabs[kGradVecWarps][3];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    GradE& Ex = tabs[warp][0];
    GradE& Ey = tabs[warp][1];
    GradE& Ez = tabs[warp][2];
    for (int h = threadIdx.x; h < grad_hb(2 * kMaxL); h += blockDim.x)
        herm[h] = herm_t(h) | (herm_u(h) << 8) | (herm_v(h) << 16);
    for (int p = blockIdx.x; p < npairs; p += gridDim.x) {
        const ShellPairDev sp = pairs[p];
        const int s1 = sp.s1, s2 = sp.s2, la = sp.l1, lb = sp.l2, L = la + lb;
        const int nc1 = ncart(la), nc2 = ncart(lb), nf1 = nfunc[s1], nf2 = nfunc[s2];
        const double* T1 = tmat + toff[s1];
        const double* T2 = tmat + toff[s2];
        const int64_t l1 = loc[s1], l2 = loc[s2];
        const double w = (s1 != s2) ? 2.0 : 1.0;
        __syncthreads();
        for (int e = threadIdx.x; e < nc1 * nc2; e += blockDim.x) {
            const int a = e / nc2, b = e - a * nc2;
            double acc = 0.0;
            for (int mb = 0; mb < nf2; ++mb) {
                double row = 0.0;
                for (int ma = 0; ma < nf1; ++ma) {
                    const int64_t pp = l1 + ma, qq = l2 + mb;
                    row += T1[ma * nc1 + a] * 0.5 * (D[pp + ldd * qq] + D[qq + ldd * pp]);
                }
                acc += row * T2[mb * nc2 + b];
            }
            Dc[e] = w * acc;
        }
        if (threadIdx.x < nc1 + nc2) {
            const int which = threadIdx.x >= nc1, c = which ? threadIdx.x - nc1 : threadIdx.x;
            const int g = cart_off(which ? lb : la) + c;
            cart[which][c] = cart_x(g) | (cart_y(g) << 8) | (cart_z(g) << 16);
        }
        __syncthreads();
        const double ax = xyz[3 * s1], ay = xyz[3 * s1 + 1], az = xyz[3 * s1 + 2];
        const double bx = xyz[3 * s2], by = xyz[3 * s2 + 1], bz = xyz[3 * s2 + 2];
        const double r2 = (ax - bx) * (ax - bx) + (ay - by) * (ay - by) + (az - bz) * (az - bz);
        const int HB = grad_hb(L);
        const int HL = herm_n(L);
        for (int i = warp; i < sp.npp; i += kGradVecWarps) {
            const int code = plist[sp.list_off + i];
            const int ga = code & 0xff, gb = code >> 8;
            const double ea = exps[poff[s1] + ga], eb = exps[poff[s2] + gb];
            const double ca = coefs[poff[s1] + ga], cb = coefs[poff[s2] + gb];
            const double P = ea + eb;
            const double px = (ea * ax + eb * bx) / P, py = (ea * ay + eb * by) / P, pz = (ea * az + eb * bz) / P;
            const double K = exp(-ea * eb / P * r2) * ca * cb;
            const double h = 1.0 / (2.0 * P);
            __syncwarp();   // the previous primitive pair's readers are done
            double* tz = &tabs[warp][0].e[0][0][0];
            for (int e = lane; e < 3 * GradE::NI * GradE::NI * GradE::NT; e += 32) tz[e] = 0.0;
            __syncwarp();
            if (lane < 3) {
                const double pc = lane == 0 ? px : (lane == 1 ? py : pz);
                const double ac = lane == 0 ? ax : (lane == 1 ? ay : az), bc = lane == 0 ? bx : (lane == 1 ? by : bz);
                grad_etab(tabs[warp][lane], la, lb, pc - ac, pc - bc, h);
            }
            __syncwarp();
            const int64_t g = gbase[p] + i;
            const int64_t li = g - level_beg[L];
            const int64_t nL = level_n[L];
            double* vg = vecs + vec_off[L] + li * (int64_t)(kGradVec * HB);
            // entry (t, u, v) of the seven vectors: every nonzero product lies within one unit above
            // the pair's range on each axis, and within level L + 1 in total
            for (int hh = lane; hh < HB; hh += 32) {
                const int t = herm[hh] & 255, u = (herm[hh] >> 8) & 255, v = herm[hh] >> 16;
                double s[kGradVec] = {};
                for (int a = 0; a < nc1; ++a) {
                    const int A = cart[0][a], axx = A & 255, ayy = (A >> 8) & 255, azz = A >> 16;
                    for (int b = 0; b < nc2; ++b) {
                        const double d = K * Dc[a * nc2 + b];
                        const int B = cart[1][b], bxx = B & 255, byy = (B >> 8) & 255, bzz = B >> 16;
                        if (d == 0.0 || t > axx + bxx + 1 || u > ayy + byy + 1 || v > azz + bzz + 1) continue;
                        const double z0 = Ez.e[azz][bzz][v];
                        const double zA = 2.0 * ea * Ez.e[azz + 1][bzz][v] - (azz > 0 ? azz * Ez.e[azz - 1][bzz][v] : 0.0);
                        const double zB = 2.0 * eb * Ez.e[azz][bzz + 1][v] - (bzz > 0 ? bzz * Ez.e[azz][bzz - 1][v] : 0.0);
                        const double y0 = Ey.e[ayy][byy][u];
                        const double yA = 2.0 * ea * Ey.e[ayy + 1][byy][u] - (ayy > 0 ? ayy * Ey.e[ayy - 1][byy][u] : 0.0);
                        const double yB = 2.0 * eb * Ey.e[ayy][byy + 1][u] - (byy > 0 ? byy * Ey.e[ayy][byy - 1][u] : 0.0);
                        const double x0 = Ex.e[axx][bxx][t];
                        const double xA = 2.0 * ea * Ex.e[axx + 1][bxx][t] - (axx > 0 ? axx * Ex.e[axx - 1][bxx][t] : 0.0);
                        const double xB = 2.0 * eb * Ex.e[axx][bxx + 1][t] - (bxx > 0 ? bxx * Ex.e[axx][bxx - 1][t] : 0.0);
                        s[0] += d * x0 * y0 * z0;
                        s[1] += d * xA * y0 * z0;
                        s[2] += d * x0 * yA * z0;
                        s[3] += d * x0 * y0 * zA;
                        s[4] += d * xB * y0 * z0;
                        s[5] += d * x0 * yB * z0;
                        s[6] += d * x0 * y0 * zB;
                    }
                }
#pragma unroll
                for (int c = 0; c < kGradVec; ++c) vg[c * HB + hh] = s[c];
                // ket role: (-1)^{tau+nu+phi} h(tau), transposed within the level
                if (hh < HL) hk[hk_off[L] + (int64_t)hh * nL + li] = ((t + u + v) & 1) ? -s[0] : s[0];
            }
            if (lane == 0) {
                mP[g] = P; mX[g] = px; mY[g] = py; mZ[g] = pz;
                ppair[g] = p;
            }
        }
    }
}

// One warp per primitive pair: the seven dot products of its vectors with its
// potential, out[g * 7 + c] (c = 0: h.V, 1..3: gA.V, 4..6: gB.V); the lanes read
// consecutive entries (one read of the vectors: bound by HBM).  Where the chunks
// left parts of the potential, each lane first adds up those of its entries, in
// their order: a call's bits then do not depend on the order in which the classes
// ran.  All levels in one launch: at 42 AOs (up to 26 parts an entry) 10 us, the
// latency of the reads (16 us with the vectors read after the parts and eight parts
// in flight), where a launch a level took 20 on potentials that came summed.
__global__ void k_grad_dots(const GradDotsArgs a)
{
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t g = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); g < a.n; g += warps) {
        int L = 0;
        while (L < kGradMaxL && g >= a.beg[L + 1]) ++L;
        const int HB = grad_hb(L);
        const int64_t i = g - a.beg[L];
        const double* vg = a.vecs + a.vec_off[L] + i * (int64_t)(kGradVec * HB);
        double* vi = a.V + a.pot_off[L] + i * (int64_t)HB;
        double s[kGradVec] = {};
        for (int h = lane; h < HB; h += 32) {
            double w[kGradVec], v = 0.0;
#pragma unroll
            for (int c = 0; c < kGradVec; ++c) w[c] = __ldg(vg + c * HB + h);
            if (a.part) {
                const double* p = a.part + a.part_off[L] + i * (int64_t)HB + h;
                const int64_t len = a.len[L];
                const int slots = a.slots[L];
#pragma unroll 16
                for (int q = 0; q < slots; ++q) v += __ldg(p + q * len);
                vi[h] = v;
            } else {
                v = vi[h];
            }
#pragma unroll
            for (int c = 0; c < kGradVec; ++c) s[c] = fma(w[c], v, s[c]);
        }
#pragma unroll
        for (int c = 0; c < kGradVec; ++c) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s[c] += __shfl_xor_sync(0xffffffffu, s[c], o);
            if (lane == c) a.out[g * kGradVec + c] = s[c];
        }
    }
}

// Coulomb matrix J_pq = sum_rs (pq|rs) Ds_rs: one block per shell pair; a
// few threads per Cartesian pair (a, b) contract the pair's primitive-pair
// records (K c_a c_b and the Hermite products E^{ab}_tuv, as the ERI kernels
// read them) with the potentials, each every few primitive pairs, then the
// block applies the two shells' transforms and writes the (s1, s2) block and its
// transpose.
constexpr int kGradMatThreads = 256;
__global__ void __launch_bounds__(kGradMatThreads) k_grad_coulomb_matrix(const ShellPairDev* __restrict__ pairs, int npairs,
                                      const int64_t* __restrict__ gbase, const int* __restrict__ level_beg,
                                      const int64_t* __restrict__ pot_off, const double* __restrict__ V,
                                      const double* __restrict__ pp, const double* __restrict__ tmat,
                                      const int* __restrict__ toff, const int* __restrict__ nfunc,
                                      const int* __restrict__ loc, double* __restrict__ J, int64_t ldj)
{
    __shared__ double Jc[ncart(kMaxL) * ncart(kMaxL)];
    __shared__ double Jh[ncart(kMaxL) * ncart(kMaxL)];
    __shared__ int ext[ncart(kMaxL) * ncart(kMaxL)];   // Hermite extent of every Cartesian pair
    __shared__ double part[kGradMatThreads];
    for (int p = blockIdx.x; p < npairs; p += gridDim.x) {
        const ShellPairDev sp = pairs[p];
        const int s1 = sp.s1, s2 = sp.s2, la = sp.l1, lb = sp.l2, L = la + lb;
        const int nc1 = ncart(la), nc2 = ncart(lb), nf1 = nfunc[s1], nf2 = nfunc[s2];
        const int HB = grad_hb(L);
        const int rs = pp_record(la, lb), po = pp_prod_off(la, lb);
        __syncthreads();
        for (int e = threadIdx.x; e < nc1 * nc2; e += blockDim.x) ext[e] = pair_x(la, lb, e) | (pair_y(la, lb, e) << 8) | (pair_z(la, lb, e) << 16);
        __syncthreads();
        const int nE = nc1 * nc2, per = kGradMatThreads / nE;   // threads per Cartesian pair (nE <= 100)
        if (threadIdx.x < per * nE) {
            const int e = threadIdx.x % nE;
            int off = 0;
            for (int f = 0; f < e; ++f) off += ((ext[f] & 255) + 1) * (((ext[f] >> 8) & 255) + 1) * ((ext[f] >> 16) + 1);
            const int ex = ext[e] & 255, ey = (ext[e] >> 8) & 255, ez = ext[e] >> 16;
            double acc = 0.0;
            for (int i = threadIdx.x / nE; i < sp.npp; i += per) {
                const double* rec = pp + sp.rec_off + (int64_t)i * rs;
                const double* prod = rec + po + off;
                const int64_t g = gbase[p] + i;
                const double* vi = V + pot_off[L] + (g - level_beg[L]) * (int64_t)HB;
                double s = 0.0;
                int c = 0;
                for (int v = 0; v <= ez; ++v)
                    for (int u = 0; u <= ey; ++u)
                        for (int t = 0; t <= ex; ++t) s += prod[c++] * vi[herm_idx(t, u, v)];
                acc += rec[4] * s;
            }
            part[threadIdx.x] = acc;
        }
        __syncthreads();
        for (int e = threadIdx.x; e < nE; e += blockDim.x) {
            double acc = 0.0;
            for (int q = 0; q < per; ++q) acc += part[q * nE + e];
            Jc[e] = acc;
        }
        __syncthreads();
        const double* T1 = tmat + __ldg(toff + s1);
        const double* T2 = tmat + __ldg(toff + s2);
        for (int e = threadIdx.x; e < nf1 * nc2; e += blockDim.x) {
            const int ma = e / nc2, b = e - ma * nc2;
            double acc = 0.0;
            for (int a = 0; a < nc1; ++a) acc += T1[ma * nc1 + a] * Jc[a * nc2 + b];
            Jh[e] = acc;
        }
        __syncthreads();
        const int64_t l1 = loc[s1], l2 = loc[s2];
        for (int e = threadIdx.x; e < nf1 * nf2; e += blockDim.x) {
            const int ma = e / nf2, mb = e - ma * nf2;
            // a shell with itself: (ma, mb) and (mb, ma) differ in their last bits, one of them counts
            if (s1 == s2 && ma < mb) continue;
            double acc = 0.0;
            for (int b = 0; b < nc2; ++b) acc += Jh[ma * nc2 + b] * T2[mb * nc2 + b];
            J[(l1 + ma) + ldj * (l2 + mb)] = acc;
            J[(l2 + mb) + ldj * (l1 + ma)] = acc;
        }
    }
}

static GradLaunchFn g_grad_launch[kGradMaxL + 1][kGradMaxL + 1];

cudaError_t grad_module_init()
{
    // the table is filled once; concurrent first calls wait for it
    static std::once_flag once;
    std::call_once(once, [] {
        register_grad_pot_a(g_grad_launch);
        register_grad_pot_b(g_grad_launch);
        register_grad_pot_c(g_grad_launch);
    });
    return cudaSuccess;
}

cudaError_t grad_pair_vectors_launch(const ShellPairDev* pairs, int npairs, const int64_t* gbase,
                                     const int* level_beg, const int* level_n, const int64_t* vec_off,
                                     const int64_t* hk_off, const double* xyz, const int* poff, const double* exps,
                                     const double* coefs, const int* plist, const double* tmat, const int* toff,
                                     const int* nfunc, const int* loc, const double* D, int64_t ldd, double* mP,
                                     double* mX, double* mY, double* mZ, double* vecs, double* hk, int* ppair,
                                     cudaStream_t st)
{
    if (npairs <= 0) return cudaSuccess;
    const int blocks = npairs < 148 * 32 ? npairs : 148 * 32;
    k_grad_pair_vectors<<<blocks, 32 * kGradVecWarps, 0, st>>>(pairs, npairs, gbase, level_beg, level_n, vec_off, hk_off, xyz, poff,
                                               exps, coefs, plist, tmat, toff, nfunc, loc, D, ldd, mP, mX, mY, mZ,
                                               vecs, hk, ppair);
    count_launch();
    return cudaGetLastError();
}

cudaError_t grad_potential_launch(int L1, int L2, const GradPotArgs& a, cudaStream_t st)
{
    if (L1 < 0 || L2 < 0 || L1 > kGradMaxL || L2 > kGradMaxL || !g_grad_launch[L1][L2]) return cudaErrorInvalidValue;
    if (a.nbra <= 0 || a.nket <= 0) return cudaSuccess;
    g_grad_launch[L1][L2](a, st);
    count_launch();
    return cudaGetLastError();
}

cudaError_t grad_dots_launch(const GradDotsArgs& a, cudaStream_t st)
{
    if (a.n <= 0) return cudaSuccess;
    int64_t blocks = (a.n + 3) / 4;
    if (blocks > 148 * 16) blocks = 148 * 16;
    k_grad_dots<<<(unsigned)blocks, 128, 0, st>>>(a);
    count_launch();
    return cudaGetLastError();
}

cudaError_t grad_coulomb_matrix_launch(const ShellPairDev* pairs, int npairs, const int64_t* gbase,
                                       const int* level_beg, const int64_t* pot_off, const double* V, const double* pp,
                                       const double* tmat, const int* toff, const int* nfunc, const int* loc,
                                       double* J, int64_t ldj, cudaStream_t st)
{
    if (npairs <= 0) return cudaSuccess;
    const int blocks = npairs < 148 * 32 ? npairs : 148 * 32;
    k_grad_coulomb_matrix<<<blocks, kGradMatThreads, 0, st>>>(pairs, npairs, gbase, level_beg, pot_off, V, pp, tmat, toff, nfunc,
                                                  loc, J, ldj);
    count_launch();
    return cudaGetLastError();
}

} // namespace gci
