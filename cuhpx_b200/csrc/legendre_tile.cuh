// FP32 Legendre contractions of many maps on CUDA cores: 128 columns (64 maps).
//
// With tens of maps the products are the work: every Pbar value meets 128
// columns, 64 packed FMAs.  A CTA is 8 multiplying warps, 2 generating and 2
// loading ones (384 threads, one CTA an SM: the 64 sums, the fragments and their
// addresses want more than the 112 registers that two CTAs would leave).
//
//   generators  run the FP64 recurrences (lane = ring; two operations a value,
//               normalised as in legendre_direct.cuh) and write FP32 values into
//               one of four shared-memory stages;
//   loaders     bring the stage's data operand by cp.async;
//   multipliers four warps per parity of l - m (the fold makes the two parities
//               independent sums), 8 x 8 results a thread: per step 4 16-byte
//               shared loads, 8 register copies (Pbar into both halves of a pair) and
//               32 packed FMAs, so the FMA pipe (a packed FMA every second clock
//               and scheduler) is the bound, not issue or shared memory.
//
// The stages change hands through named barriers.
// Measured (nside 512, L = M = 1023, 64 maps): analysis contraction 4109 -> 3026 us
// (the kernel that generated and multiplied in the same threads), synthesis 5694
// -> 2843 us (that kernel; 5016 us by the direct one), 55% of the FMA rate: what
// is left is the exposed latency of two multiplying warps a scheduler and
// the padding of 128-degree blocks.  Blocks at the end of an order leave out the
// warps that have no degrees, and the analysis' loaders keep the next stage's rows in
// flight while they hand one over (whole call of that size 4189 -> 4157 us, nside
// 256, L = 511 825 -> 806 us; either alone changes nothing).
#pragma once

#include "legendre_direct.cuh"

namespace hpx {

constexpr int kTileCols = 128;
constexpr int kTileMul = 256, kTileGen = 64, kTileLoad = 64;  // threads of each kind
constexpr int kTileThreads = kTileMul + kTileGen + kTileLoad;
constexpr int kTileStages = 4;

// stage s handed over (all threads of one side arrive, those of the other wait)
__device__ __forceinline__ void tile_arrive(int id) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(kTileThreads) : "memory"); }
__device__ __forceinline__ void tile_wait(int id) { asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(kTileThreads) : "memory"); }
__device__ __forceinline__ int tile_full(int s) { return 1 + s; }
__device__ __forceinline__ int tile_empty(int s) { return 1 + kTileStages + s; }

// n steps acc[i][j] += p[i] * x[j] (8 values by 4 column pairs) from p and x on,
// PS and XS floats a step (unrolled by 2 / 4 / 8: nside 512, 64 maps, analysis
// 3625 / 3095 / 3026 us -- the loads of the next steps hide behind the FMAs only
// within one unrolled body)
template <int PS, int XS>
__device__ __forceinline__ void tile_steps(Pair<float> (&acc)[8][4], const float* p, const float* x, int n) {
#pragma unroll 8
    for (int k = 0; k < n; ++k) {
        Pair<float> x0[2], x1[2];
        load_pairs<2>(x0, x + k * XS);
        load_pairs<2>(x1, x + k * XS + 64);
        const float4 pa = *(const float4*)(p + k * PS), pb = *(const float4*)(p + k * PS + 4);
        const float pv[8] = {pa.x, pa.y, pa.z, pa.w, pb.x, pb.y, pb.z, pb.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const Pair<float> pp = Pair<float>::make(pv[i], pv[i]);
            acc[i][0].fma(pp, x0[0]);
            acc[i][1].fma(pp, x0[1]);
            acc[i][2].fma(pp, x1[0]);
            acc[i][3].fma(pp, x1[1]);
        }
    }
}

// ------------------------------------------------------------ analysis
constexpr int kTileDeg = 128;                     // degrees per CTA: two seed blocks
constexpr int kTileRing = 32;                     // rings per stage
constexpr int kTilePRow = kTileDeg + 4;           // [even 64][odd 64], padded: 16-byte stores of 8 lanes on distinct banks
constexpr int kTileFwdStage = kTileRing * kTilePRow + kTileRing * 2 * kTileCols;  // floats
constexpr size_t kTileFwdSmem = (size_t)kTileStages * kTileFwdStage * sizeof(float);

// alm[b][l][m] (+)= sum_p Pbar_l^m(z_p) X[m][par][p][2b..] (X: k_fold's spec, C
// columns), 128 columns from 128 blockIdx.y on.  CTA x < ntiles: four orders by nj degree blocks, order fastest, so that
// neighbouring CTAs complete the same 32-byte sectors of alm and share X[m] in L2;
// CTAs x >= ntiles clear the m > l entries.
__global__ void __launch_bounds__(kTileThreads, 1)
    k_leg_fwd_tile(const float* __restrict__ spec, int C, int nmaps, float* __restrict__ alm, int L, int M, Geom geo,
                   const double* __restrict__ z, const int* __restrict__ lstart, const double2* __restrict__ pstart,
                   const double* __restrict__ alpha, const double2* __restrict__ norm, int Lpad,
                   const double2* __restrict__ seeds, int nj, int ntiles, int accumulate) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_first;
    float* stages = (float*)smem_raw;
    const int tid = threadIdx.x, NP = geo.NP;
    const int c0 = blockIdx.y * kTileCols, b0 = c0 / 2;  // first column and map
    if ((int)blockIdx.x >= ntiles) {
        // a warp per row and map (by whole CTAs, 64 maps one after the other, the rows
        // took 30 us of 421 at nside 64, L = 127, 512 maps a pass)
        const int nb = min(kTileCols / 2, nmaps - b0), lane = tid & 31;
        for (int l = blockIdx.x - ntiles; l < min(L, M - 1); l += gridDim.x - ntiles)
            for (int b = b0 + (tid >> 5); b < b0 + nb; b += kTileThreads / 32) {
                cplx<float>* row = (cplx<float>*)alm + ((int64_t)b * L + l) * M;
                for (int m = l + 1 + lane; m < M; m += 32)
                    if (HPX_INB(2 * (((int64_t)b * L + l) * M + m) + 1, kExtAlm, 15)) row[m] = {0.f, 0.f};
            }
        return;
    }
    const int r4 = blockIdx.x % (4 * nj);
    const int m = blockIdx.x / (4 * nj) * 4 + (r4 & 3), l0 = m + (r4 >> 2) * kTileDeg;
    if (m >= M || l0 >= L) return;
    const int t0 = geo.first_ring(m);
    // first ring with a value above 2^-1000 among these degrees (the rings before it
    // hold zeros)
    if (tid == 0) s_first = NP;
    __syncthreads();
    int first = NP;
    for (int p = t0 + tid; p < NP; p += kTileThreads)
        if (lstart[(int64_t)m * NP + p] < min(l0 + kTileDeg, L)) {
            first = p;
            break;
        }
    first = __reduce_min_sync(0xffffffffu, first);
    if ((tid & 31) == 0 && first < NP) atomicMin(&s_first, first);
    __syncthreads();
    const int p0 = s_first;
    const int nch = (NP - p0 + kTileRing - 1) / kTileRing;
    const int64_t mo = (int64_t)m * Lpad;

    if (tid >= kTileMul) {
        if (tid >= kTileMul + kTileGen) {
            // ------------------------------------------------ loaders: 32 lanes = the 512 bytes of a row
            const int lane = tid & 31, par = (tid >> 5) & 1;
            for (int c = 0; c < nch; ++c) {
                const int st = c % kTileStages, pc = p0 + c * kTileRing, nr = min(kTileRing, NP - pc);
                float* Xs = stages + st * kTileFwdStage + kTileRing * kTilePRow + par * kTileCols + 4 * lane;
                if (c >= kTileStages) tile_wait(tile_empty(st));
                const float* src = spec + (((int64_t)m * 2 + par) * NP + pc) * C + c0 + 4 * lane;
                if (c0 + 4 * lane < C) {  // (columns past C are never written out)
#pragma unroll 8
                    for (int q = 0; q < nr; ++q)
                        if (HPX_INB(src + (int64_t)q * C + 3 - spec, kExtSpec, 29))
                            cp_async16(Xs + 2 * q * kTileCols, src + (int64_t)q * C);
                }
                cp_async_commit();
                if (c > 0) {  // hand over the stage before; this one's rows stay in flight
                    cp_async_wait<1>();
                    tile_arrive(tile_full((c - 1) % kTileStages));
                }
            }
            cp_async_wait<0>();
            if (nch > 0) tile_arrive(tile_full((nch - 1) % kTileStages));
            return;
        }
        // ---------------------------------------------------- generators: lane = ring, warp = block of 64 degrees
        const int g = tid - kTileMul, lane = g & 31, half = g >> 5;
        const int lb = l0 + 64 * half;
        const double* al = alpha + mo + 2 + lb;
        const double2* nm = norm + mo;
        const double2* sp = seeds + ((int64_t)m * seed_blocks(L) + (lb - m) / kSeedBlock) * NP;
        if (lb >= L) {  // no degree of the order, and nobody reads the values
            for (int c = 0; c < nch; ++c) {
                if (c >= kTileStages) tile_wait(tile_empty(c % kTileStages));
                tile_arrive(tile_full(c % kTileStages));
            }
            return;
        }
        const double n0 = nm[lb].y, n1 = lb + 1 < L ? nm[lb + 1].y : 0.0;
        // a ring's start degree, node and seeds, fetched a stage ahead
        int ls_n = kNoDegree;
        double x_n = 0.0;
        double2 sd_n = make_double2(0.0, 0.0);
        auto fetch = [&](int c) {
            const int p = p0 + c * kTileRing + lane;
            ls_n = kNoDegree;
            if (p < NP) {
                ls_n = lstart[(int64_t)m * NP + p];
                x_n = z[p];
                sd_n = sp[p];
            }
        };
        if (nch > 0) fetch(0);
        for (int c = 0; c < nch; ++c) {
            const int st = c % kTileStages, p = p0 + c * kTileRing + lane;
            float* row = stages + st * kTileFwdStage + lane * kTilePRow + 32 * half;
            const int ls = ls_n < L ? ls_n : kNoDegree;
            const double x = x_n;
            double u0 = 0.0, u1 = 0.0;
            if (ls <= lb) {
                u0 = sd_n.x * n0;
                u1 = sd_n.y * n1;
            }
            if (c + 1 < nch) fetch(c + 1);
            const bool late = __any_sync(0xffffffffu, ls > lb && ls < lb + 64);  // some ring starts in here
            if (c >= kTileStages) tile_wait(tile_empty(st));
            double an[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) an[k] = al[k];
            // (a start test between the steps would serialise them: 125 clocks a
            // step instead of about 35)
            auto run = [&](auto starts) {
#pragma unroll 1
                for (int i = 0; i < 64; i += 8) {
                    float v[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const double a = an[k];
                        an[k] = al[i + 8 + k];  // eight degrees ahead
                        if constexpr (decltype(starts)::value) {
                            if (ls == lb + i + k && i + k > 0) {
                                const double2 ps = dir_start<float>(pstart[(int64_t)m * NP + p], nm, ls, L);
                                u0 = ps.x;
                                u1 = ps.y;
                            }
                        }
                        v[k] = (float)u0;
                        DirRec<float>::advance(a, x, u0, u1);
                    }
                    *(float4*)(row + i / 2) = make_float4(v[0], v[2], v[4], v[6]);
                    *(float4*)(row + 64 + i / 2) = make_float4(v[1], v[3], v[5], v[7]);
                }
            };
            if (late) run(DirYes{});
            else run(DirNo{});
            tile_arrive(tile_full(st));
        }
        return;
    }
    // -------------------------------------------------------- multipliers
    const int par = tid >> 7, tx = tid & 15, ty = (tid >> 4) & 7;
    const bool rows = l0 + 16 * (ty & ~1) + par < L;  // the warp (two ty) has degrees of the order
    Pair<float> acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = Pair<float>::zero();
    for (int c = 0; c < nch; ++c) {
        const int st = c % kTileStages;
        const float* Ps = stages + st * kTileFwdStage + 64 * par + 8 * ty;
        const float* Xs = stages + st * kTileFwdStage + kTileRing * kTilePRow + par * kTileCols + 4 * tx;
        tile_wait(tile_full(st));
        if (rows) tile_steps<kTilePRow, 2 * kTileCols>(acc, Ps, Xs, min(kTileRing, NP - p0 - c * kTileRing));
        if (c + kTileStages < nch) tile_arrive(tile_empty(st));
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int l = l0 + 2 * (8 * ty + i) + par;
        if (l >= L) continue;
        const double cn = norm[mo + l].x;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int b = b0 + 2 * tx + (j & 1) + (j >> 1) * 32;
            const int64_t o = ((int64_t)b * L + l) * M + m;
            if (b >= nmaps || !HPX_INB(2 * o + 1, kExtAlm, 16)) continue;
            const float2 q = acc[i][j].get();
            cplx<float> v = {(float)((double)q.x * cn), (float)((double)q.y * cn)};
            cplx<float>* dst = (cplx<float>*)alm + o;
            if (accumulate) v = cadd(*dst, v);
            *dst = v;
        }
    }
}

// ------------------------------------------------------------ synthesis
constexpr int kTileInvRing = 64;  // rings per CTA
constexpr int kTileInvDeg = 64;   // degrees per stage
constexpr int kTileInvStage = kTileInvDeg * kTileInvRing + kTileInvDeg * kTileCols;  // floats
constexpr size_t kTileInvSmem = (size_t)kTileStages * kTileInvStage * sizeof(float);

// alm[b][l][m] -> almT[m][l][C] = a_lm c_l, columns 2b + {re, im} (zeros past
// nmaps).  CTA: 32 orders x one degree, 256 threads, 64 maps from 64 blockIdx.z on.
__global__ void __launch_bounds__(256) k_alm_to_tile(const float* __restrict__ alm, int nmaps, int L, int M,
                                                     const double2* __restrict__ norm, int Lpad,
                                                     float* __restrict__ almT, int C) {
    __shared__ cplx<float> tile[64][33];
    const int m0 = blockIdx.x * 32, l = blockIdx.y, b0 = blockIdx.z * 64;
    if (m0 > l) return;  // only m <= l is read
    const int tid = threadIdx.x, tx = tid & 31;
    const int m = m0 + tx;
    const double c = m <= l && m < M ? norm[(int64_t)m * Lpad + l].x : 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int b = b0 + (tid >> 5) + 8 * k;
        cplx<float> v = {0.f, 0.f};
        const int64_t o = ((int64_t)b * L + l) * M + m;
        if (b < nmaps && m <= l && m < M && HPX_INB(2 * o + 1, kExtAlm, 27)) v = ((const cplx<float>*)alm)[o];
        tile[b - b0][tx] = {(float)((double)v.re * c), (float)((double)v.im * c)};
    }
    __syncthreads();
    // one warp writes an order's 128 columns as 16-byte pieces
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int i = (tid >> 5) + 8 * k, mm = m0 + i;
        if (mm > l || mm >= M || 2 * b0 + 4 * tx >= C) continue;
        const cplx<float> a = tile[2 * tx][i], b = tile[2 * tx + 1][i];
        const int64_t o = ((int64_t)mm * L + l) * C + 2 * b0 + 4 * tx;
        if (HPX_INB(o + 3, kExtAlmT, 31)) *(float4*)(almT + o) = make_float4(a.re, a.im, b.re, b.im);
    }
}

// spec[m][0|1][p][C]: sums over l - m even | odd for order m = blockIdx.y and rings
// 64 blockIdx.x .. + 64, 128 columns from 128 blockIdx.z on (unfold and the inverse ring FFTs follow)
__global__ void __launch_bounds__(kTileThreads, 1)
    k_leg_inv_tile(const float* __restrict__ almT, int C, float* __restrict__ spec, int L, int M, Geom geo,
                   const double* __restrict__ z, const int* __restrict__ lstart, const double2* __restrict__ pstart,
                   const double* __restrict__ alpha, const double2* __restrict__ norm, int Lpad) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_first;
    float* stages = (float*)smem_raw;
    const int tid = threadIdx.x, NP = geo.NP;
    const int m = blockIdx.y, pb = blockIdx.x * kTileInvRing, c0 = blockIdx.z * kTileCols;
    const int t0 = geo.first_ring(m);
    if (pb + kTileInvRing <= t0) return;
    if (tid == 0) s_first = L;
    __syncthreads();
    if (tid < kTileInvRing) {
        const int p = pb + tid;
        if (p >= t0 && p < NP && m < L) atomicMin(&s_first, lstart[(int64_t)m * NP + p]);
    }
    __syncthreads();
    const int lbeg = m + (max(s_first - m, 0) & ~(kTileInvDeg - 1));  // whole stages of zeros are skipped
    const int nch = s_first < L ? (L - lbeg + kTileInvDeg - 1) / kTileInvDeg : 0;

    if (tid >= kTileMul) {
        if (tid >= kTileMul + kTileGen) {
            const int lane = tid & 31, w = (tid >> 5) & 1;  // loaders: a warp per degree of either parity
            for (int c = 0; c < nch; ++c) {
                const int st = c % kTileStages, lc = lbeg + c * kTileInvDeg, nl = min(kTileInvDeg, L - lc);
                float* As = stages + st * kTileInvStage + kTileInvDeg * kTileInvRing + 4 * lane;
                if (c >= kTileStages) tile_wait(tile_empty(st));
                const float* src = almT + ((int64_t)m * L + lc) * C + c0 + 4 * lane;
                if (c0 + 4 * lane < C) {
#pragma unroll 8
                    for (int i = w; i < nl; i += 2)
                        if (HPX_INB(src + (int64_t)i * C + 3 - almT, kExtAlmT, 30))
                            cp_async16(As + i * kTileCols, src + (int64_t)i * C);
                }
                cp_async_commit();
                cp_async_wait<0>();
                tile_arrive(tile_full(st));
            }
            return;
        }
        const int g = tid - kTileMul, p = pb + g;  // generators: a ring each
        const double* al = alpha + (int64_t)m * Lpad + 2;
        const double2* nm = norm + (int64_t)m * Lpad;
        double x = 0.0, u0 = 0.0, u1 = 0.0;
        int ls = kNoDegree;
        if (p >= t0 && p < NP && m < L) {
            const int s = lstart[(int64_t)m * NP + p];
            if (s < L) ls = s;
            x = z[p];
        }
        double an[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) an[k] = nch > 0 ? al[lbeg + k] : 0.0;
        for (int c = 0; c < nch; ++c) {
            const int st = c % kTileStages, lc = lbeg + c * kTileInvDeg;
            float* Ps = stages + st * kTileInvStage + g;
            const bool late = __any_sync(0xffffffffu, ls >= lc && ls < lc + kTileInvDeg);  // some ring starts in here
            if (c >= kTileStages) tile_wait(tile_empty(st));
            auto run = [&](auto starts) {
#pragma unroll 1
                for (int i = 0; i < kTileInvDeg; i += 8) {
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const double a = an[k];
                        an[k] = al[lc + i + 8 + k];  // eight degrees ahead
                        if constexpr (decltype(starts)::value) {
                            if (ls == lc + i + k) {
                                const double2 ps = dir_start<float>(pstart[(int64_t)m * NP + p], nm, ls, L);
                                u0 = ps.x;
                                u1 = ps.y;
                            }
                        }
                        Ps[(i + k) * kTileInvRing] = (float)u0;
                        DirRec<float>::advance(a, x, u0, u1);
                    }
                }
            };
            if (late) run(DirYes{});
            else run(DirNo{});
            tile_arrive(tile_full(st));
        }
        return;
    }
    const int par = tid >> 7, tx = tid & 15, ty = (tid >> 4) & 7;
    Pair<float> acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = Pair<float>::zero();
    for (int c = 0; c < nch; ++c) {
        const int st = c % kTileStages;
        const float* Ps = stages + st * kTileInvStage + par * kTileInvRing + 8 * ty;
        const float* As = stages + st * kTileInvStage + kTileInvDeg * kTileInvRing + par * kTileCols + 4 * tx;
        tile_wait(tile_full(st));
        const int nl = min(kTileInvDeg, L - lbeg - c * kTileInvDeg), nk = (nl - par + 1) >> 1;  // this parity's degrees
        if (nk > 0) tile_steps<2 * kTileInvRing, 2 * kTileCols>(acc, Ps, As, nk);
        if (c + kTileStages < nch) tile_arrive(tile_empty(st));
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int p = pb + 8 * ty + i;
        const int64_t o = (((int64_t)m * 2 + par) * NP + p) * C + c0;
        if (p < t0 || p >= NP || !HPX_INB(o + min(kTileCols, C - c0) - 1, kExtSpec, 28)) continue;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (c0 + 64 * h + 4 * tx >= C) continue;
            const float2 a = acc[i][2 * h].get(), b = acc[i][2 * h + 1].get();
            *(float4*)(spec + o + 64 * h + 4 * tx) = make_float4(a.x, a.y, b.x, b.y);
        }
    }
}

}  // namespace hpx
