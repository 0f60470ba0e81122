// eri_hermite.cuh -- product-mode ERI stages in Hermite-matrix form on the
// FP64 tensor-core path (DMMA, mma.sync m8n8k4 f64).
//
// For a row shell pair AB (primitive pairs i) and a column shell pair CD
// (primitive pairs k), every (ab|cd) of the McMurchie-Davidson sum of the
// reference (auto2e_WMatrix_part1.f90:743-812, Hermite recursions of
// auto2e_Hermite.f90) is
//     (r|J) = sum_i sum_h Er_i(r, h) sum_k sum_g R_ik(h + g) Ec_k(g, J)
// where r runs over the (spherical, normalised) functions of the row pair,
// J over the requested functions of the column pair, and
//     Er_i(r, h) = K_ab c_a c_b sum_{a,b} T_A(r_a, a) T_B(r_b, b) E^{ab}_i(h)
//     Ec_k(g, J) = (-1)^|g| K_cd c_c c_d sum_{c,d} T_C(J_c, c) T_D(J_d, d) E^{cd}_k(g)
// are the pair's Hermite vectors (E^{ab} the two-centre Hermite coefficients
// of the primitive pair, T the normalisation x solid-harmonic transforms).
// The Cartesian -> spherical transforms of the reference
// (auto2e_SpherTransf.f90, auto2e_Normalize_*) are thus applied to the
// Hermite coefficients once per primitive pair instead of to every
// contracted quartet, and the ket side carries only the columns a stage
// keeps (pivot columns in the full-dimension stage, Step2.f90:242-419).
//
// Row primitive pairs are taken in blocks of IB and column primitive pairs in
// groups of KP, so that the products have no padding between primitive pairs:
//     X((i,h), J) += sum_{(k,g)} R_ik(h + g) Ec((k,g), J)
// over the IB H1 rows of a block and the KP H2 columns of a group, then
//     O(r, J) += sum_{(i,h)} Er(r, (i,h)) X((i,h), J)
// per block.  One warp evaluates one (row pair, column chunk) task.
//
// The R_tuv of a batch of primitive quartets are evaluated one quartet per
// lane (or per SL lanes), entirely in registers (hm_quartet), and left in
// warp-private shared memory; the products then gather their Hankel operand from there through a
// table of byte offsets, one 16-byte table load per eight fragments.  A unit is
// one (block, group) combination of IB KP quartets; a batch holds UB of them.
//
// Bound by the FP64 tensor pipe where tasks are many (12 atoms of s4p3d2f1 with
// 3-6 primitives, 4912 vectors: step-1 columns 1477 -> 830 ms, full-dimension
// stage 1269 -> 648 ms against a form that took one primitive quartet at a time,
// built its R level by level with 32 lanes in shared memory between the tensor
// instructions, and padded every primitive pair to whole tiles).  Warps: 12 an SM
// at 168 registers while the accumulators are few, else 8 with up to 255.
#pragma once
#include "gci_common.h"
#include "boys.cuh"
#include <algorithm>
#include <atomic>
#include <type_traits>

namespace gci {

template <int L1, int L2, int NT>
struct HmShape {
    static constexpr int LT = L1 + L2;
    static constexpr int H1 = herm_n(L1), H2 = herm_n(L2), HT = herm_n(LT);
    static constexpr int IB = hm_ib(L1), KP = hm_kp(L2), UQ = IB * KP;
    static constexpr int MT = hm_mt(L1), KT = hm_kt(L2), MTO = hm_mto(L1);
    static constexpr int RSTR = hm_row_stride(L1), CSTR = hm_col_stride(L2, NT);
    static constexpr int TILES = MT * NT;
    // 4 warps a block; 3 blocks an SM (168 registers a thread) while the accumulators are few
    static constexpr int WARPS = 4, TPB = 32 * WARPS, MINB = TILES <= 12 ? 3 : 2;
    // doubles of a quartet's R in the batch: odd, so that lanes storing the same entry of
    // consecutive quartets fall into different banks
    static constexpr int QS = HT | 1;
    // ring of column fragments: PD k-steps, copied PD - 1 steps ahead
    static constexpr int PD = TILES >= 8 ? 4 : 8;
    static constexpr int RING = PD * NT * 32;
    static constexpr int OS = MTO * 8 * NT * 8;   // output block O(r, J), fragment order [MTO][NT][32][2]
    // table of byte offsets: [KT][32][MTP] 16-bit entries
    static constexpr int MTP = MT <= 2 ? 2 : (MT <= 4 ? 4 : (MT + 3) / 4 * 4);
    static constexpr int TAB = KT * 32 * MTP;   // shorts
    // units of a batch: at most 32 quartets (one per lane) within the warp's share of 227 KB
    static constexpr int BUDGET = ((MINB == 3 ? 74 : 112) * 1024 - 2 * TAB) / (8 * WARPS) - RING - OS;   // doubles
    static constexpr int UB_MEM = BUDGET / (UQ * QS), UB_LANE = UQ >= 32 ? 1 : 32 / UQ;
    static constexpr int UB = UB_MEM < 1 ? 1 : (UB_MEM < UB_LANE ? UB_MEM : UB_LANE);
    static constexpr int RSZ = (UB * UQ * QS + 1) & ~1;
    // lanes per quartet of the R recursion
    static constexpr int SL = UB * UQ * 4 <= 32 && LT >= 4 ? 4 : (UB * UQ * 2 <= 32 && LT >= 2 ? 2 : 1);
    static constexpr int WS = RSZ + RING + OS;
    // the next k-step's Hankel fragments are loaded one step ahead (registers: 2 MT)
    static constexpr bool APF = MT <= 7;
    static constexpr size_t smem_bytes() { return sizeof(double) * (size_t)WARPS * WS + sizeof(short) * (size_t)TAB; }
    static_assert(UQ * QS * 8 <= 65535, "unit offsets are 16-bit");
    static_assert(sizeof(double) * (size_t)WARPS * WS + 2 * TAB <= 227 * 1024, "shared memory");
};

template <int I, int N, class Fn>
__device__ __forceinline__ void hm_static_for(Fn&& fn)
{
    if constexpr (I < N) {
        fn(std::integral_constant<int, I>{});
        hm_static_for<I + 1, N>(fn);
    }
}

// D = A B + D for one 8x8x4 tile: lane l holds A[l/4][l%4], B[l%4][l/4] and
// D[l/4][2(l%4) + {0,1}].
__device__ __forceinline__ void dmma884(double (&d)[2], double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
        : "+d"(d[0]), "+d"(d[1])
        : "d"(a), "d"(b));
}

// One step of the Hermite Coulomb recursion along one axis (Helgaker 9.9.18-20)
// for all orders n at fixed other components:
//   R^{(n)}_{c} = d R^{(n+1)}_{c-1} + (c - 1) R^{(n+1)}_{c-2},  n = 0 .. M - c
// from p1 = R_{c-1} (orders 0..M-c+1) and p2 = R_{c-2}; result over p2.
template <int M, int C, int N1, int N2>
__device__ __forceinline__ void hm_axis_step(double d, const double (&p1)[N1], double (&p2)[N2])
{
#pragma unroll
    for (int n = 0; n <= M - C; ++n) p2[n] = C > 1 ? fma((double)(C - 1), p2[n + 1], d * p1[n + 1]) : d * p1[n + 1];
}

// R_tuv = R^{(0)}_tuv, t+u+v <= LT, of one primitive quartet from
// F^{(n)} = (-2 alpha)^n pref F_n, stored at out[hm_ridx(LT,t,u,v)].  The levels
// are walked axis by axis: the order-n row of R_{00v} gives the rows R_{0uv},
// and those the R_{tuv}, so only two rows per axis are live (a level-by-level
// recursion holds all herm_n(LT) values).  The same number of operations.
// S lanes share a quartet when a batch holds fewer than 32: lane s takes the
// planes v = S j + s, all lanes running the code of plane S j (its orders
// beyond a lane's plane are not stored): 2.2 to 2.4 times fewer instructions
// per quartet at S = 4.
template <int LT, int S>
__device__ __forceinline__ void hm_quartet(double (&F)[LT + 1], double X, double Y, double Z, int s,
                                           double* __restrict__ out)
{
    double a0[LT + 1], a1[LT + 1];   // rows v - 1 (or v - 2 before the step) and v
#pragma unroll
    for (int n = 0; n <= LT; ++n) a1[n] = F[n];
    hm_static_for<0, LT / S + 1>([&](auto J) {
        constexpr int v0 = decltype(J)::value * S, MV = LT - v0;
        double b0[MV + 1], b1[MV + 1];
        hm_static_for<0, (S < MV + 1 ? S : MV + 1)>([&](auto W) {
            constexpr int v = v0 + decltype(W)::value;
            if constexpr (v == 1) {
#pragma unroll
                for (int n = 0; n <= LT; ++n) a0[n] = a1[n];
                hm_axis_step<LT, 1>(Z, a0, a1);
            } else if constexpr (v > 1) {
                // a1 holds v - 1, a0 holds v - 2
                hm_axis_step<LT, v>(Z, a1, a0);
#pragma unroll
                for (int n = 0; n <= LT; ++n) { const double t = a0[n]; a0[n] = a1[n]; a1[n] = t; }
            }
            if constexpr (v == v0) {
#pragma unroll
                for (int n = 0; n <= MV; ++n) b1[n] = a1[n];
            } else {
#pragma unroll
                for (int n = 0; n <= LT - v; ++n) b1[n] = s == v - v0 ? a1[n] : b1[n];
            }
        });
        const int vl = v0 + s;   // this lane's plane
        double* __restrict__ pl = out + hm_ridx(LT, 0, 0, vl <= LT ? vl : LT);
        hm_static_for<0, MV + 1>([&](auto U) {
            constexpr int u = decltype(U)::value, MU = MV - u;
            if constexpr (u == 1) {
#pragma unroll
                for (int n = 0; n <= MV; ++n) b0[n] = b1[n];
                hm_axis_step<MV, 1>(Y, b0, b1);
            } else if constexpr (u > 1) {
                hm_axis_step<MV, u>(Y, b1, b0);
#pragma unroll
                for (int n = 0; n <= MV; ++n) { const double t = b0[n]; b0[n] = b1[n]; b1[n] = t; }
            }
            double c0[MU + 1], c1[MU + 1];
#pragma unroll
            for (int n = 0; n <= MU; ++n) c1[n] = b1[n];
            hm_static_for<0, MU + 1>([&](auto T) {
                constexpr int t = decltype(T)::value;
                if constexpr (t == 1) {
#pragma unroll
                    for (int n = 0; n <= MU; ++n) c0[n] = c1[n];
                    hm_axis_step<MU, 1>(X, c0, c1);
                } else if constexpr (t > 1) {
                    hm_axis_step<MU, t>(X, c1, c0);
#pragma unroll
                    for (int n = 0; n <= MU; ++n) { const double w = c0[n]; c0[n] = c1[n]; c1[n] = w; }
                }
                // planes v0 + s with LT - v0 - s < t + u do not have this entry
                if (S == 1 || t + u <= MV - (S - 1) || s <= MV - t - u) pl[hm_ridx(LT, t, u, 0)] = c1[0];
            });
        });
    });
}

// R of the primitive quartet (row primitive record Bp, column primitive record Kp),
// all zero when !on (padding of a unit); s: this lane's share of the S.  One
// function per level and split, called once per lane and batch.
template <int LT, int S>
__device__ __noinline__ void hm_produce(const double* __restrict__ Bp, const double* __restrict__ Kp, double kappa,
                                        const double* __restrict__ boys, int on, int s, double* __restrict__ out)
{
    const double P = __ldg(Bp), Q = __ldg(Kp);
    const double dx = __ldg(Bp + 1) - __ldg(Kp + 1), dy = __ldg(Bp + 2) - __ldg(Kp + 2), dz = __ldg(Bp + 3) - __ldg(Kp + 3);
    // Boys values scaled by the quartet's factor and (-2 alpha)^m
    double alpha, pref;
    quartet_factors(P, Q, kappa, alpha, pref);
    double F[LT + 1];
    boys_fm<LT>(alpha * (dx * dx + dy * dy + dz * dz), boys, F);
    double pw = on ? pref : 0.0;
    const double m2a = -2.0 * alpha;
#pragma unroll
    for (int m = 0; m <= LT; ++m) { F[m] *= pw; pw *= m2a; }
    hm_quartet<LT, S>(F, dx, dy, dz, s, out);
}

// 8-byte asynchronous copy global -> shared
__device__ __forceinline__ void hm_cp8(uint32_t dst, const double* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}

// table words of one lane and k-step: MTP 16-bit byte offsets
template <int MTP>
struct HmIdx {
    uint32_t w[MTP / 2];
    __device__ __forceinline__ void load(const unsigned short* p)
    {
        if constexpr (MTP == 2) {
            w[0] = *reinterpret_cast<const uint32_t*>(p);
        } else if constexpr (MTP % 8 == 0) {
#pragma unroll
            for (int q = 0; q < MTP / 8; ++q) {
                const uint4 v = reinterpret_cast<const uint4*>(p)[q];
                w[4 * q] = v.x; w[4 * q + 1] = v.y; w[4 * q + 2] = v.z; w[4 * q + 3] = v.w;
            }
        } else {
#pragma unroll
            for (int q = 0; q < MTP / 4; ++q) {
                const uint2 v = reinterpret_cast<const uint2*>(p)[q];
                w[2 * q] = v.x; w[2 * q + 1] = v.y;
            }
        }
    }
    __device__ __forceinline__ uint32_t get(int m) const { return (m & 1) ? w[m >> 1] >> 16 : w[m >> 1] & 0xffffu; }
};

template <int L1, int L2, int NT>
__global__ void __launch_bounds__(HmShape<L1, L2, NT>::TPB, HmShape<L1, L2, NT>::MINB)
k_eri_hm(const HmArgs a)
{
    using S = HmShape<L1, L2, NT>;
    constexpr int LT = S::LT, MT = S::MT, KT = S::KT, MTO = S::MTO, IB = S::IB, KP = S::KP, UQ = S::UQ, UB = S::UB;
    constexpr int PD = S::PD;
    extern __shared__ __align__(16) double smem[];
    unsigned short* tab = reinterpret_cast<unsigned short*>(smem + (size_t)S::WARPS * S::WS);

    // Hankel fragment (m, ks) of a unit: lane l reads R_{il,kl}(h + g) with (il, h) = 8 m + l/4 and
    // (kl, g) = 4 ks + l%4 flattened over the unit's rows and columns.  Padding reads entry 0 (a
    // finite value): its column vectors or its row vectors are zero.
    // (t | u << 8 | v << 16 of the Hermite indices first, where the warps' data will be)
    int* herm = reinterpret_cast<int*>(smem);
    constexpr int HMAX = S::H1 > S::H2 ? S::H1 : S::H2;
    static_assert(HMAX * sizeof(int) <= sizeof(double) * S::WARPS * S::WS, "index list");
    for (int h = threadIdx.x; h < HMAX; h += S::TPB) herm[h] = herm_t(h) | (herm_u(h) << 8) | (herm_v(h) << 16);
    __syncthreads();
    for (int c = threadIdx.x; c < S::TAB; c += S::TPB) {
        const int m = c % S::MTP, l = (c / S::MTP) & 31, ks = c / (S::MTP * 32);
        const int rho = 8 * m + (l >> 2), kap = 4 * ks + (l & 3);
        int off = 0;
        if (rho < IB * S::H1 && kap < KP * S::H2) {
            const int il = rho / S::H1, h = rho - il * S::H1, kl = kap / S::H2, g = kap - kl * S::H2;
            const int tuv = herm[h] + herm[g];   // no carries: components stay below 256
            off = 8 * ((il * KP + kl) * S::QS + hm_ridx(LT, tuv & 255, (tuv >> 8) & 255, tuv >> 16));
        }
        tab[c] = (unsigned short)off;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double* Rb = smem + (size_t)warp * S::WS;
    double* ring = Rb + S::RSZ + lane;
    double* Os = Rb + S::RSZ + S::RING;
    const uint32_t ring_s = (uint32_t)__cvta_generic_to_shared(ring);
    __syncthreads();

    const int64_t nparts = a.nrows * a.nchunks * a.split;
    for (;;) {
        // tasks in row-major order (a row pair's chunks are consecutive), taken
        // one (or one part) at a time from the launch's counter
        unsigned long long t0 = 0;
        if (lane == 0) t0 = atomicAdd(a.counter, 1ULL);
        const int64_t tpart = (int64_t)__shfl_sync(0xffffffffu, t0, 0);
        if (tpart >= nparts) break;
        const int64_t task = tpart / a.split;
        const int part = (int)(tpart - task * a.split);
        const int64_t rix = task / a.nchunks;
        const HmChunk ch = a.chunks[a.chunk_ids[task - rix * a.nchunks]];
        const int rp = a.rows[rix];
        if (a.upper && ch.pair < rp) continue;   // the mirror image of another task
        const ShellPairDev pr = a.pairs[rp];
        const ShellPairDev pc = a.pairs[ch.pair];
        const int nb = pr.npp, nk = pc.npp;
        const int nib = (nb + IB - 1) / IB, nkg = (nk + KP - 1) / KP;
        const int ib0 = nib * part / a.split, nu = (nib * (part + 1) / a.split - ib0) * nkg;
        const int rsr = pp_record(pr.l1, pr.l2), rsc = pp_record(pc.l1, pc.l2);
        const double* __restrict__ rrec = a.pp + pr.rec_off;
        const double* __restrict__ crec = a.pp + pc.rec_off;
        const double* __restrict__ rowv = a.rowvec + a.rowvec_off[rp];
        const double* __restrict__ colv = a.colvec + ch.vec_off + lane;
        const double* const colv_end = colv + (size_t)nkg * S::CSTR;
        const int first = pr.swap ? pr.s2 : pr.s1, second = pr.swap ? pr.s1 : pr.s2;
        const int n1 = __ldg(a.sh_nfunc + first);
        const int nR = n1 * __ldg(a.sh_nfunc + second);

        // each lane owns entries 2 lane + {0,1} of every 64-entry tile of the block
        for (int w = 2 * lane; w < S::OS; w += 64) { Os[w] = 0.0; Os[w + 1] = 0.0; }

        // the column fragments of all units in order, PD - 1 k-steps ahead (each lane copies and
        // reads its own elements); every block of rows runs through the same column vectors
        const double* cpf = colv;
        uint32_t slot_w = 0, slot_r = 0;
        auto prefetch = [&]() {
#pragma unroll
            for (int n = 0; n < NT; ++n) hm_cp8(ring_s + 8 * (slot_w * NT + n) * 32, cpf + n * 32);
            asm volatile("cp.async.commit_group;" ::: "memory");
            slot_w = (slot_w + 1) & (PD - 1);
            cpf += NT * 32;
            if (cpf == colv_end) cpf = colv;
        };
        if (nu > 0) {
#pragma unroll
            for (int s = 0; s < PD - 1; ++s) prefetch();
        }

        double X[MT][NT][2];
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int n = 0; n < NT; ++n) X[m][n][0] = X[m][n][1] = 0.0;
        int ib = ib0, kg = 0;   // block and group of the unit whose products come next

        for (int u0 = 0; u0 < nu; u0 += UB) {
            const int un = nu - u0 < UB ? nu - u0 : UB;
            __syncwarp();
            // R of the batch, one quartet per SL lanes
#pragma unroll 1
            for (int q = lane / S::SL; q < un * UQ; q += 32 / S::SL) {
                const int ul = q / UQ, rq = q - ul * UQ;
                const int u = u0 + ul, uib = u / nkg, ukg = u - uib * nkg;
                int i = (ib0 + uib) * IB + rq / KP, k = ukg * KP + rq % KP;
                const int on = i < nb && k < nk;
                if (!on) i = k = 0;
                hm_produce<LT, S::SL>(rrec + (size_t)i * rsr, crec + (size_t)k * rsc, a.kappa, a.boys, on,
                                      lane % S::SL, Rb + q * S::QS);
            }
            __syncwarp();
            const char* Ru = reinterpret_cast<const char*>(Rb);
            for (int ul = 0; ul < un; ++ul) {
                // rows of the block in use: whole tiles of its primitive pairs (blocks of one pair are full)
                const int mte = (IB == 1 || (ib + 1) * IB <= nb) ? MT : ((nb - ib * IB) * S::H1 + 7) / 8;
                const char* const Rn = ul + 1 < un ? Ru + UQ * S::QS * 8 : Ru;
                auto steps = [&](auto FULL) {
                    constexpr bool full = decltype(FULL)::value;
                    const unsigned short* tp = tab + lane * S::MTP;
                    double rn[S::APF ? MT : 1];
                    if constexpr (S::APF) {
                        HmIdx<S::MTP> ix;
                        ix.load(tp);
#pragma unroll
                        for (int m = 0; m < MT; ++m) rn[m] = *reinterpret_cast<const double*>(Ru + ix.get(m));
                    }
#pragma unroll 1
                    for (int ks = 0; ks < KT; ++ks) {
                        asm volatile("cp.async.wait_group %0;" ::"n"(PD - 2) : "memory");
                        double e[NT];
#pragma unroll
                        for (int n = 0; n < NT; ++n) e[n] = ring[(slot_r * NT + n) * 32];
                        slot_r = (slot_r + 1) & (PD - 1);
                        prefetch();
                        if constexpr (S::APF) {
                            double r[MT];
#pragma unroll
                            for (int m = 0; m < MT; ++m) r[m] = rn[m];
                            tp += 32 * S::MTP;
                            if (ks + 1 < KT) {
                                HmIdx<S::MTP> ix;
                                ix.load(tp);
#pragma unroll
                                for (int m = 0; m < MT; ++m) rn[m] = *reinterpret_cast<const double*>(Ru + ix.get(m));
                            }
#pragma unroll
                            for (int m = 0; m < MT; ++m) {
                                if (full || m < mte) {
#pragma unroll
                                    for (int n = 0; n < NT; ++n) dmma884(X[m][n], e[n], r[m]);
                                }
                            }
                        } else {
                            HmIdx<S::MTP> ix;
                            ix.load(tp);
                            tp += 32 * S::MTP;
#pragma unroll
                            for (int m = 0; m < MT; ++m) {
                                const double r = *reinterpret_cast<const double*>(Ru + ix.get(m));
#pragma unroll
                                for (int n = 0; n < NT; ++n) dmma884(X[m][n], e[n], r);
                            }
                        }
                    }
                };
                if (IB == 1 || mte == MT) steps(std::true_type{});
                else steps(std::false_type{});
                Ru = Rn;
                if (++kg < nkg) continue;
                // O(r, J) += Er(r, (i,h)) X((i,h), J): the accumulator element e of tile m holds row
                // 8 m + 2 (l%4) + e of X at column J = l/4, which is a B fragment of k-step 2 m + e
                // with the row vectors in that order
                const double* __restrict__ rv = rowv + (size_t)ib * S::RSTR + lane;
                constexpr int MO = NT >= 4 ? 1 : (NT >= 2 ? 2 : (MTO < 4 ? MTO : 4));   // output tiles at once
#pragma unroll 1
                for (int m0 = 0; m0 < MTO; m0 += MO) {
                    if (8 * m0 >= nR) break;
                    double acc[MO][NT][2];
#pragma unroll
                    for (int o = 0; o < MO; ++o)
#pragma unroll
                        for (int n = 0; n < NT; ++n) acc[o][n][0] = acc[o][n][1] = 0.0;
#pragma unroll
                    for (int ks = 0; ks < 2 * MT; ++ks)
#pragma unroll
                        for (int o = 0; o < MO; ++o) {
                            if (MTO % MO != 0 && m0 + o >= MTO) continue;
                            const double av = __ldg(rv + ((m0 + o) * 2 * MT + ks) * 32);
#pragma unroll
                            for (int n = 0; n < NT; ++n) dmma884(acc[o][n], av, X[ks >> 1][n][ks & 1]);
                        }
#pragma unroll
                    for (int o = 0; o < MO; ++o) {
                        if (MTO % MO != 0 && m0 + o >= MTO) continue;
                        double2* od = reinterpret_cast<double2*>(Os + (m0 + o) * NT * 64 + 2 * lane);
#pragma unroll
                        for (int n = 0; n < NT; ++n) {
                            double2 w = od[n * 32];
                            w.x += acc[o][n][0];
                            w.y += acc[o][n][1];
                            od[n * 32] = w;
                        }
                    }
                }
#pragma unroll
                for (int m = 0; m < MT; ++m)
#pragma unroll
                    for (int n = 0; n < NT; ++n) X[m][n][0] = X[m][n][1] = 0.0;
                kg = 0;
                ++ib;
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");

        if (a.split > 1) {
            const int used = (nR + 7) / 8 * NT * 64;
            double* pt = a.part + task * a.split * S::OS;
            if (nu > 0)
                for (int w = 2 * lane; w < used; w += 64)
                    __stcg(reinterpret_cast<double2*>(pt + part * S::OS + w), *reinterpret_cast<const double2*>(Os + w));
            __threadfence();
            __syncwarp();
            int last = 0;
            if (lane == 0) last = atomicAdd(a.arrive + task, 1) == a.split - 1;
            if (!__shfl_sync(0xffffffffu, last, 0)) continue;
            __threadfence();
            for (int w = 2 * lane; w < used; w += 64) {
                double2 sum = make_double2(0.0, 0.0);
                for (int q = 0; q < a.split; ++q) {
                    // a part without blocks, or a task without column primitive pairs, left nothing
                    if (nkg == 0 || nib * q / a.split == nib * (q + 1) / a.split) continue;
                    const double2 v = __ldcg(reinterpret_cast<const double2*>(pt + q * S::OS + w));
                    sum.x += v.x;
                    sum.y += v.y;
                }
                *reinterpret_cast<double2*>(Os + w) = sum;
            }
        }

        // scatter: element (m, n, l, e) of the block is O(8 m + l/4, 8 n + 2 (l%4) + e)
#pragma unroll 1
        for (int m = 0; m < MTO; ++m) {
            const int r = 8 * m + (lane >> 2);
            if (r >= nR) continue;
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int J = 8 * n + 2 * (lane & 3) + e;
                    if (J >= ch.ncol) continue;
                    const int col = a.colout[ch.col_off + J];
                    if (col < 0) continue;
                    const double val = Os[(m * NT + n) * 64 + 2 * lane + e];
                    if (a.mode == kModeProduct) {
                        const int row = a.row_map[a.row_off[rp] + r];
                        if (row >= 0) a.out[row + a.ldo * (int64_t)col] = val;
                    } else {
                        const int i1 = r % n1, i2 = r / n1;
                        const int64_t p = __ldg(a.sh_loc + first) + i1, q = __ldg(a.sh_loc + second) + i2;
                        a.out[(p * a.nao + q) * a.jcount + col] = val;
                        if (first != second) a.out[(q * a.nao + p) * a.jcount + col] = val;
                    }
                }
        }
    }
}

} // namespace gci

namespace gci {

// How a class is launched: warps resident at once on the device (0: a CUDA error), doubles of
// a task's output block, and the launch itself.
struct HmLaunch {
    cudaError_t (*launch)(const HmArgs&, cudaStream_t);
    int (*resident)();
    int block;
};

// The shared-memory attribute is set on every launch: it belongs to the
// current device, and the library may be called on several devices.
template <int L1, int L2, int NT>
static cudaError_t hm_prepare()
{
    return cudaFuncSetAttribute(k_eri_hm<L1, L2, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)HmShape<L1, L2, NT>::smem_bytes());
}

// Blocks resident at once: a property of the kernel and of the sm_100a GPU it is built for, the
// same on every device, so it is asked once.
template <int L1, int L2, int NT>
static int hm_resident_blocks()
{
    using S = HmShape<L1, L2, NT>;
    static std::atomic<int> known{0};
    int n = known.load(std::memory_order_relaxed);
    if (n > 0) return n;
    int dev = 0, nsm = 0, per_sm = 0;
    if (hm_prepare<L1, L2, NT>() != cudaSuccess || cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_eri_hm<L1, L2, NT>, S::TPB, S::smem_bytes()) !=
            cudaSuccess)
        return 0;
    n = nsm * (per_sm < 1 ? 1 : per_sm);
    known.store(n, std::memory_order_relaxed);
    return n;
}

template <int L1, int L2, int NT>
static int hm_resident()
{
    return hm_resident_blocks<L1, L2, NT>() * HmShape<L1, L2, NT>::WARPS;
}

template <int L1, int L2, int NT>
static cudaError_t launch_hm(const HmArgs& a, cudaStream_t st)
{
    using S = HmShape<L1, L2, NT>;
    const int64_t nparts = a.nrows * a.nchunks * a.split;
    if (nparts <= 0) return cudaSuccess;
    cudaError_t e = hm_prepare<L1, L2, NT>();
    if (e != cudaSuccess) return e;
    // persistent: as many blocks as are resident at once; warps take tasks from a.counter
    const int64_t cap = hm_resident_blocks<L1, L2, NT>();
    if (cap <= 0) return cudaErrorInvalidDevice;
    const int64_t blocks = std::min<int64_t>((nparts + S::WARPS - 1) / S::WARPS, cap);
    k_eri_hm<L1, L2, NT><<<(unsigned)blocks, S::TPB, S::smem_bytes(), st>>>(a);
    return cudaGetLastError();
}

// tab[L1][L2][NT - 1] for L2 = 0 .. kMaxPairL and NT = 1 .. hm_max_nt(L1)
template <int L1, int L2, int NT = 1>
static void register_hm_nt(HmLaunch (*tab)[kMaxPairL + 1][kHmMaxNT])
{
    tab[L1][L2][NT - 1] = {&launch_hm<L1, L2, NT>, &hm_resident<L1, L2, NT>, HmShape<L1, L2, NT>::OS};
    if constexpr (NT < hm_max_nt(L1)) register_hm_nt<L1, L2, NT + 1>(tab);
}

template <int L1, int L2 = 0>
static void register_hm_row(HmLaunch (*tab)[kMaxPairL + 1][kHmMaxNT])
{
    register_hm_nt<L1, L2>(tab);
    if constexpr (L2 < kMaxPairL) register_hm_row<L1, L2 + 1>(tab);
}

void register_hm_0(HmLaunch (*tab)[kMaxPairL + 1][kHmMaxNT]);
void register_hm_1(HmLaunch (*tab)[kMaxPairL + 1][kHmMaxNT]);
void register_hm_2(HmLaunch (*tab)[kMaxPairL + 1][kHmMaxNT]);
void register_hm_3(HmLaunch (*tab)[kMaxPairL + 1][kHmMaxNT]);
void register_hm_4(HmLaunch (*tab)[kMaxPairL + 1][kHmMaxNT]);
void register_hm_5(HmLaunch (*tab)[kMaxPairL + 1][kHmMaxNT]);
void register_hm_6(HmLaunch (*tab)[kMaxPairL + 1][kHmMaxNT]);

} // namespace gci
