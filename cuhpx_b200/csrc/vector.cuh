// Spin-1 (vector) Legendre contractions on CUDA cores, FP32 or FP64.
//
// cuHPX's VectorSHT / VectoriSHT (cuhpx/hpx_sht.py:286-444) transform a
// tangent field given as two real components [batch][2][npix] into
// spheroidal and toroidal coefficients [batch][2][L][M] with the table
// _precompute_dlegpoly (cuhpx/sht_tools.py:267-304), for 0 <= m <= l:
//   D0_l^m = 0.5 (sqrt((l+m)(l-m+1)) Pbar_l^{m-1} - sqrt((l-m)(l+m+1)) Pbar_l^{m+1})
//            (Pbar_l^{-1} := -Pbar_l^1, so D0_l^0 = -sqrt(l(l+1)) Pbar_l^1)
//   D1_l^m = 0.5 sqrt((2l+1)/(2l+3)) (sqrt((l-m+1)(l-m+2)) Pbar_{l+1}^{m-1}
//            + sqrt((l+m+1)(l+m+2)) Pbar_{l+1}^{m+1}),   D1_l^0 = 0
// times (-1)^m when csphase is set.  With the folded ring spectra x0, x1 of the
// two components (quadrature weights included) and nf_l = 1/(l(l+1)), nf_0 = 1:
//   S_lm = nf_l sum_t (D0 x0 - i D1 x1)       T_lm = nf_l sum_t (-D0 x1 - i D1 x0)
// and the synthesis of ring spectra (s, t) of the two components:
//   s_tm = sum_l (D0 S + i D1 T)              t_tm = sum_l (-D0 T + i D1 S).
// The reference tabulates D0, D1 densely ([2][M][L][rings], FP64) and runs
// eight einsums per call.  Here they are generated on the fly:
//
//   FP32  from the one recurrence of order m that the scalar kernels run: D0 is
//         dPbar/dtheta and D1 is m Pbar / sin(theta), so
//           sin(theta) D0_l = f_l Pbar_{l+1} - (l+1) x Pbar_l,
//           f_l = sqrt((2l+1)/(2l+3) ((l+1)^2 - m^2)),    sin(theta) D1_l = m Pbar_l
//         with the pair (Pbar_l, Pbar_{l+1}) the recurrence carries anyway;
//         1/sin(theta) goes into the folded spectra or onto the finished ring
//         sums.  The subtraction, in FP64, loses a factor 1/sin(theta) next to
//         the poles: nothing FP32 values notice (errors against FP64 measured 10
//         to 40% below the form with two recurrences), but
//   FP64  would (3e-14 against 5e-15 in maps at nside 256), so it runs the
//         recurrences of orders m-1 and m+1 (two more operations a value beside the
//         16 of the products).
// The vector plan is built with L+1 degrees and M+1 orders for them.
//
// North/south symmetry: Pbar_l^m(-x) = (-1)^{l+m} Pbar_l^m(x), so D0 has the
// parity (-1)^{l+m+1} and D1 the parity (-1)^{l+m}: the analysis contracts D0
// with the fold of parity index (l-m+1)&1 and D1 with (l-m)&1 (S = w(F_t +
// F_t'), D = w(F_t - F_t')); the synthesis sums the terms whose south sign is +
// into E and the others into O (F_t = E + O, F_t' = E - O).  The two components
// of every vector map travel through the ring FFTs as two consecutive maps.
//
// The kernels are those of legendre_direct.cuh with two values and eight columns
// per vector map: a warp per order, 32 R rings by lane, nothing tabulated and no
// fold or unfold launch.  The tiled kernels before
// them ran recurrences of orders m-1 and m+1 and 64 columns whatever the batch:
// analysis + synthesis of 4 maps at nside 128, L = M = 255, FP32 1282 -> 158 us.
#pragma once

#include "legendre_direct.cuh"

namespace hpx {

// Factors of degree l: FP32 f_l c_{l+1} / c_l and l + 1; FP64 those of the four
// terms of D0 and D1
template <typename T>
struct VecFac;
template <>
struct VecFac<float> {
    double f, lp;
    static __device__ __forceinline__ VecFac make(int l, int m, const double2* __restrict__ nm, int Lv) {
        if (l >= Lv) return {0.0, 0.0};
        const double dl = l;
        const double f = sqrt((2.0 * dl + 1.0) / (2.0 * dl + 3.0) * ((dl + 1.0 - m) * (dl + 1.0 + m)));
        return {f * nm[l + 1].x * nm[l].y, dl + 1.0};
    }
};
template <>
struct VecFac<double> {
    double c1, c2, c3, c4;
    static __device__ __forceinline__ VecFac make(int l, int m, const double2* __restrict__, int Lv) {
        if (l >= Lv || l < m) return {0.0, 0.0, 0.0, 0.0};
        const double dl = l, dm = m;
        const double h = 0.5 * sqrt((2.0 * dl + 1.0) / (2.0 * dl + 3.0));
        return {0.5 * sqrt((dl + dm) * (dl - dm + 1.0)), 0.5 * sqrt((dl - dm) * (dl + dm + 1.0)),
                m ? h * sqrt((dl - dm + 1.0) * (dl - dm + 2.0)) : 0.0, m ? h * sqrt((dl + dm + 1.0) * (dl + dm + 2.0)) : 0.0};
    }
};

// One ring's generator at degree l: the values p0 ~ D0_l, p1 ~ D1_l (FP32: times
// sin(theta) / c_l, and 1 / m for p1).  start(l) must be called before value() at
// every degree at which a recurrence may start.
template <typename T>
struct VecGen;
template <>
struct VecGen<float> {
    static constexpr bool kScaled = true;  // 1/sin(theta) and m are applied elsewhere
    int ls;
    double x, u0, u1;
    struct Order {
        const double* coef;  // alpha of degree l + 2 at [l]
        const double2* nm;
        int64_t row;  // m * NP
        int m, L;
    };
    static __device__ __forceinline__ Order order(int m, int, int Lp, int Lpad, int NP, const double* coef,
                                                  const double2* norm) {
        return {coef + (int64_t)m * Lpad + 2, norm + (int64_t)m * Lpad, (int64_t)m * NP, m, Lp};
    }
    __device__ __forceinline__ void clear() {
        ls = kNoDegree;
        x = u0 = u1 = 0.0;
    }
    // first degree (from l0 on) that can be nonzero, kNoDegree if none below lend
    __device__ __forceinline__ int init(const Order& o, int p, double z, int l0, int lend,
                                        const int* __restrict__ lstart) {
        x = z;
        const int s = lstart[o.row + p];
        if (s < lend) ls = s;
        return ls;
    }
    // the pair at l0 (= m + a multiple of 64) from the block seeds
    __device__ __forceinline__ void seed(const Order& o, int p, int NP, int l0, const double2* __restrict__ seeds,
                                         const double2* __restrict__) {
        if (ls <= l0) {
            const double2 sd =
                dir_start<float>(seeds[((int64_t)o.m * seed_blocks(o.L) + (l0 - o.m) / kSeedBlock) * NP + p], o.nm, l0, o.L);
            u0 = sd.x;
            u1 = sd.y;
            ls = l0 - 1;  // started
        }
    }
    __device__ __forceinline__ int last_start(int l0) const { return ls >= l0 && ls < kNoDegree ? ls : -1; }
    __device__ __forceinline__ void start(const Order& o, int p, int l, const double2* __restrict__ pstart) {
        if (ls == l) {
            const double2 ps = dir_start<float>(pstart[o.row + p], o.nm, l, o.L);
            u0 = ps.x;
            u1 = ps.y;
        }
    }
    struct Coef {
        double al;
    };
    static __device__ __forceinline__ Coef load(const Order& o, int l) { return {o.coef[l]}; }
    __device__ __forceinline__ void value(const VecFac<float>& f, int, float& p0, float& p1) const {
        p0 = (float)fma(f.f, u1, -(f.lp * x) * u0);
        p1 = (float)u0;
    }
    __device__ __forceinline__ void advance(const Coef& c) { DirRec<float>::advance(c.al, x, u0, u1); }
};
template <>
struct VecGen<double> {
    static constexpr bool kScaled = false;
    int la, lb;                   // starts of orders m - 1 and m + 1
    double x, a0, a1, b0, b1;     // their pairs at l, l + 1
    struct Order {
        const double2 *ca, *cb;
        int64_t ra, rb;
        int m, L;
    };
    static __device__ __forceinline__ Order order(int m, int Mp, int Lp, int Lpad, int NP, const double2* coef,
                                                  const double2*) {
        const int ma = m ? m - 1 : 0, mb = min(m + 1, Mp - 1);  // (m < Mv = Mp - 1 wherever values are used)
        return {coef + (int64_t)ma * Lpad + 2, coef + (int64_t)mb * Lpad + 2, (int64_t)ma * NP, (int64_t)mb * NP, m, Lp};
    }
    __device__ __forceinline__ void clear() {
        la = lb = kNoDegree;
        x = a0 = a1 = b0 = b1 = 0.0;
    }
    __device__ __forceinline__ int init(const Order& o, int p, double z, int l0, int lend,
                                        const int* __restrict__ lstart) {
        x = z;
        // a value of degree l also takes the pairs' second elements: one degree earlier
        const int sb = lstart[o.rb + p];
        if (sb <= lend) lb = sb;
        if (o.m) {
            const int sa = lstart[o.ra + p];
            if (sa <= lend) la = sa;
        }
        const int s = min(la, lb);
        return s == kNoDegree ? s : max(s - 1, l0);
    }
    __device__ __forceinline__ void seed(const Order& o, int p, int NP, int l0, const double2* __restrict__ seeds,
                                         const double2* __restrict__ pstart) {
        const int j = (l0 - o.m) / kSeedBlock, nb = seed_blocks(o.L);
        if (la < l0) {  // order m - 1: block j starts at l0 - 1
            const double2 sd = seeds[((int64_t)(o.m - 1) * nb + j) * NP + p];
            a0 = sd.x;
            a1 = sd.y;
            DirRec<double>::advance(o.ca[l0 - 1], x, a0, a1);
        }
        if (j > 0 && lb < l0) {  // order m + 1: block j - 1 starts at l0 - 63
            const int l1 = l0 + 1 - kSeedBlock;
            if (lb <= l1) {
                const double2 sd = seeds[((int64_t)(o.m + 1) * nb + j - 1) * NP + p];
                b0 = sd.x;
                b1 = sd.y;
            }
#pragma unroll 1
            for (int l = l1; l < l0; ++l) {
                if (lb == l && lb > l1) {
                    const double2 ps = pstart[o.rb + p];
                    b0 = ps.x;
                    b1 = ps.y;
                }
                DirRec<double>::advance(o.cb[l], x, b0, b1);
            }
        }
    }
    __device__ __forceinline__ int last_start(int l0) const {
        int s = -1;
        if (la >= l0 && la < kNoDegree) s = la;
        if (lb >= l0 && lb < kNoDegree) s = max(s, lb);
        return s;
    }
    __device__ __forceinline__ void start(const Order& o, int p, int l, const double2* __restrict__ pstart) {
        if (la == l) {
            const double2 ps = pstart[o.ra + p];
            a0 = ps.x;
            a1 = ps.y;
        }
        if (lb == l) {
            const double2 ps = pstart[o.rb + p];
            b0 = ps.x;
            b1 = ps.y;
        }
        // a start at l + 1 is already the second element of the pair at l
        if (la == l + 1) a1 = pstart[o.ra + p].x;
        if (lb == l + 1) b1 = pstart[o.rb + p].x;
    }
    struct Coef {
        double2 a, b;
    };
    static __device__ __forceinline__ Coef load(const Order& o, int l) { return {o.ca[l], o.cb[l]}; }
    __device__ __forceinline__ void value(const VecFac<double>& f, int m, double& p0, double& p1) const {
        p0 = fma(f.c1, m ? a0 : -b0, -(f.c2 * b0));  // Pbar^{-1} = -Pbar^1
        p1 = fma(f.c3, a1, f.c4 * b1);
    }
    __device__ __forceinline__ void advance(const Coef& c) {
        DirRec<double>::advance(c.a, x, a0, a1);
        DirRec<double>::advance(c.b, x, b0, b1);
    }
};

template <typename T, int CV, int R>
constexpr int vec_min_ctas() {
    return dir_min_ctas<T, 4 * CV, R>();
}

// ------------------------------------------------------------ analysis
template <typename T, int CV, int R>
__host__ __device__ constexpr size_t vfwd_smem_bytes(int lch) {
    return kDirWarps * (fwd_direct_xstride<T, 4 * CV, R>() * 2 * sizeof(T) + (size_t)lch * (8 * CV * sizeof(T) + sizeof(VecFac<T>)));
}

// CTA: orders m = 4 blockIdx.y + warp, degrees m + blockIdx.x lch .. + lch (lch a
// multiple of 64: a block seed), vector maps CV blockIdx.z .. + CV; blockIdx.x =
// nch clears the rows' m > l entries.  F: ring spectra of 2 nvec scalar maps;
// alm: [nvec][2][Lv][Mv] complex.  adjoint: fold factors of the synthesis' adjoint.
// use_nf = 0 leaves out the 1/(l(l+1)) factor (the adjoint of the synthesis).
template <typename T, int CV, int R>
__global__ void __launch_bounds__(32 * kDirWarps, vec_min_ctas<T, CV, R>())
    k_vleg_fwd(const T* __restrict__ F, int64_t Ftot, int nvec, T* __restrict__ alm, int Lv, int Mv, int Lp, Geom geo,
               const RingLite* __restrict__ rings, const double* __restrict__ z, const int* __restrict__ lstart,
               const double2* __restrict__ pstart, const typename DirRec<T>::Coef* __restrict__ coef,
               const double2* __restrict__ norm, int Lpad, const double2* __restrict__ seeds, int lch, int nch,
               int csphase, int adjoint, int use_nf) {
    constexpr int NC = 2 * CV;                             // complex columns
    constexpr int NV = kSumVals<T>, G = NV / (8 * CV);     // degrees per transposed sum
    static_assert(G >= 1 && (G == 1 || G % 2 == 0), "a group starts at an even l - m, or is one degree");
    constexpr int W = kDirWarps;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int NP = geo.NP;
    const int b0 = blockIdx.z * CV;
    if ((int)blockIdx.x == nch) {
        for (int l = blockIdx.y; l < min(Lv, Mv - 1); l += gridDim.y)
            for (int cc = 0; cc < NC; ++cc) {
                const int64_t row = (int64_t)(2 * b0 + cc) * Lv + l;
                if (2 * b0 + cc >= 2 * nvec) break;
                for (int m = l + 1 + threadIdx.x; m < Mv; m += blockDim.x)
                    if (HPX_INB(2 * (row * Mv + m) + 1, kExtAlm, 17)) ((cplx<T>*)alm)[row * Mv + m] = {(T)0, (T)0};
            }
        return;
    }
    constexpr size_t XS = fwd_direct_xstride<T, 4 * CV, R>();
    VecFac<T>* fac = (VecFac<T>*)smem_raw + (size_t)warp * lch;       // [W][lch]
    cplx<T>* Xs = (cplx<T>*)((VecFac<T>*)smem_raw + (size_t)W * lch);  // [W][XS]: [north, south][column][32 R rings]
    T* acc = (T*)(Xs + W * XS) + (size_t)warp * lch * 8 * CV;
    const int m0 = blockIdx.y * W, m = m0 + warp;
    const int i0 = blockIdx.x * lch, l0 = m + i0;
    if (m0 + i0 >= Lv) return;
    const bool active = m < Mv && l0 < Lv;
    const int n = active ? min(lch, Lv - l0) : 0;
    const int ng = (n + G - 1) / G;
    for (int i = lane; i < ng * NV; i += 32) acc[i] = (T)0;
    const int t0 = active ? geo.first_ring(m) : NP;
    const int64_t mo = (int64_t)min(m, Mv - 1);
    const double2* nm = norm + mo * Lpad;
    const auto ord = VecGen<T>::order((int)mo, Mv + 1, Lp, Lpad, NP, coef, norm);
    for (int i = lane; i < ng * G; i += 32) fac[i] = VecFac<T>::make(l0 + i, m, nm, Lv);

    const int perm = sum_perm<T, 2 * NC>(lane), acc_lane = (lane % (2 * G)) * 2 * NC + lane / (2 * G);
    auto stage = [&](int pb) {
#pragma unroll
        for (int kk = 0; kk < R; ++kk) {
            const int j = threadIdx.x & (W - 1), k = kk * 32 + threadIdx.x / W, p = pb + k, mj = m0 + j;
            cplx<T>* xd = Xs + j * XS + k;
            RingLite rl{};
            if (p < NP) rl = rings[p];
            const bool ok = mj < rl.mt && mj < Mv;
#pragma unroll
            for (int cc = 0; cc < NC; ++cc) {
                const int64_t fb = (int64_t)(2 * b0 + cc) * Ftot + mj;
                const bool in = ok && 2 * b0 + cc < 2 * nvec;
                if (in && HPX_INB(2 * (fb + rl.foff_n) + 1, kExtF, 25))
                    cp_async_cplx(xd + cc * 32 * R, (const cplx<T>*)F + fb + rl.foff_n);
                else
                    xd[cc * 32 * R] = {(T)0, (T)0};
                if (in && rl.foff_s >= 0 && HPX_INB(2 * (fb + rl.foff_s) + 1, kExtF, 25))
                    cp_async_cplx(xd + (NC + cc) * 32 * R, (const cplx<T>*)F + fb + rl.foff_s);
                else
                    xd[(NC + cc) * 32 * R] = {(T)0, (T)0};
            }
        }
        cp_async_commit();
    };
    const int pfirst = geo.first_ring(m0);
    if (pfirst < NP) stage(pfirst);
    for (int pb = pfirst; pb < NP; pb += 32 * R) {
        VecGen<T> gen[R];
        int lmin = kNoDegree, lmax = -1;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int p = pb + 32 * r + lane;
            gen[r].clear();
            if (p >= t0 && p < NP) {
                const int s = gen[r].init(ord, p, z[p], l0, l0 + n, lstart);
                if (s < l0 + n) {
                    gen[r].seed(ord, p, NP, l0, seeds, pstart);
                    lmin = min(lmin, s);
                    lmax = max(lmax, gen[r].last_start(l0));
                }
            }
        }
        lmin = __reduce_min_sync(0xffffffffu, lmin);
        lmax = __reduce_max_sync(0xffffffffu, lmax);
        cp_async_wait<0>();
        __syncthreads();
        Pair<T> S[R][NC], D[R][NC];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int p = min(pb + 32 * r + lane, NP - 1);
            const RingLite& rl = rings[p];
            const bool south = rl.foff_s >= 0;
            const double w0 = adjoint ? ((m == 0 || m == rl.h) ? 1.0 : 2.0) : rl.w;
            const T w = (T)(VecGen<T>::kScaled ? w0 * rl.rs : w0);  // quadrature weight (/ sin(theta))
#pragma unroll
            for (int cc = 0; cc < NC; ++cc) {
                const cplx<T>* xs = Xs + warp * XS + 32 * r + lane + (cc ^ (perm >> 1)) * 32 * R;
                const cplx<T> a = xs[0], c = xs[NC * 32 * R];
                const cplx<T> sv = cscale(cadd(a, c), w), dv = cscale(csub(a, c), south ? w : (T)0);
                S[r][cc] = perm & 1 ? Pair<T>::make(sv.im, sv.re) : Pair<T>::make(sv.re, sv.im);
                D[r][cc] = perm & 1 ? Pair<T>::make(dv.im, dv.re) : Pair<T>::make(dv.re, dv.im);
            }
        }
        __syncthreads();
        if (pb + 32 * R < NP) stage(pb + 32 * R);
        if (lmin == kNoDegree) continue;
        // one group; ODD: its first degree has l - m odd (groups of one degree)
        auto group = [&](int g, auto starts, auto odd) {
            const int lg = l0 + g * G;
            Pair<T> v[G][2][NC];
#pragma unroll
            for (int i = 0; i < G; ++i)
#pragma unroll
                for (int cc = 0; cc < NC; ++cc) v[i][0][cc] = v[i][1][cc] = Pair<T>::zero();
#pragma unroll
            for (int i = 0; i < G; ++i) {
                const auto ab = VecGen<T>::load(ord, lg + i);
                const VecFac<T> fl = fac[g * G + i];
                const bool od = ((i & 1) != 0) != decltype(odd)::value;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    if constexpr (decltype(starts)::value) gen[r].start(ord, pb + 32 * r + lane, lg + i, pstart);
                    T p0, p1;
                    gen[r].value(fl, m, p0, p1);
                    const Pair<T> pp0 = Pair<T>::make(p0, p0), pp1 = Pair<T>::make(p1, p1);
#pragma unroll
                    for (int cc = 0; cc < NC; ++cc) {
                        v[i][0][cc].fma(pp0, od ? S[r][cc] : D[r][cc]);
                        v[i][1][cc].fma(pp1, od ? D[r][cc] : S[r][cc]);
                    }
                    gen[r].advance(ab);
                }
            }
            T f[NV];
#pragma unroll
            for (int i = 0; i < G; ++i)
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int cc = 0; cc < NC; ++cc) {
                        const auto q = v[i][h][cc].get();
                        f[(2 * cc * G + i) * 2 + h] = q.x;
                        f[((2 * cc + 1) * G + i) * 2 + h] = q.y;
                    }
            const T sum = transpose_sum<T, NV, 2 * NC>(f, lane);  // lane = (column G + degree in group) 2 + h
            if (lane < NV) acc[g * NV + acc_lane] += sum;
        };
        int g = max(0, lmin - l0) / G;
        const int gs = lmax < 0 ? g : min(ng, (lmax - l0) / G + 1);
        auto run = [&](int gend, auto starts) {
            if constexpr (G == 1) {
                // l0 - m is a multiple of 64: group g has parity g & 1
                if (g < gend && (g & 1)) {
                    group(g, starts, DirYes{});
                    ++g;
                }
#pragma unroll 1
                for (; g + 1 < gend; g += 2) {
                    group(g, starts, DirNo{});
                    group(g + 1, starts, DirYes{});
                }
                if (g < gend) {
                    group(g, starts, DirNo{});
                    ++g;
                }
            } else {
#pragma unroll 1
                for (; g < gend; ++g) group(g, starts, DirNo{});
            }
        };
        run(gs, DirYes{});
        run(ng, DirNo{});
    }
    __syncwarp();
    // S = nf (A0 - i B1), T = nf (-A1 - i B0); A: D0 sums, B: D1 sums of the two components
    for (int i = lane; i < n; i += 32) {
        const int l = l0 + i;
        double c = sizeof(T) == 4 ? nm[l].x : 1.0;
        if (use_nf && l > 0) c *= 1.0 / ((double)l * (double)(l + 1));
        if (csphase && (m & 1)) c = -c;
        const double cb = VecGen<T>::kScaled ? c * m : c;
#pragma unroll
        for (int vb = 0; vb < CV; ++vb) {
            if (b0 + vb >= nvec) break;
            const cplx<T>* a = (const cplx<T>*)(acc + (size_t)i * 8 * CV) + 2 * vb;
            const cplx<T>* b = a + NC;
            const int64_t o = ((int64_t)(b0 + vb) * 2 * Lv + l) * Mv + m;
            if (!HPX_INB(2 * (o + (int64_t)Lv * Mv) + 1, kExtAlm, 18)) continue;
            ((cplx<T>*)alm)[o] = {(T)(c * a[0].re + cb * b[1].im), (T)(c * a[0].im - cb * b[1].re)};
            ((cplx<T>*)alm)[o + (int64_t)Lv * Mv] = {(T)(cb * b[0].im - c * a[1].re), (T)(-(c * a[1].im + cb * b[0].re))};
        }
    }
}

// ------------------------------------------------------------ synthesis
template <typename T, int CV, int R>
__host__ __device__ constexpr size_t vinv_smem_bytes() {
    const size_t raw = (size_t)2 * kDirWarps * kDirChunk * 2 * CV * 2 * sizeof(T);
    const size_t rows = (size_t)kDirWarps * kDirChunk * (8 * CV * sizeof(T) + sizeof(VecFac<T>));
    const size_t f = (size_t)2 * kDirWarps * 32 * R * 4 * CV * sizeof(T);
    return raw + rows > f ? raw + rows : f;
}

// CTA: orders m = 4 blockIdx.y + warp < Mp, rings 32 R blockIdx.x .. + 32 R, vector
// maps CV blockIdx.z .. + CV (as k_leg_inv_direct).  Orders the coefficients do not
// carry get zero spectra.  use_nf = 1 first scales the coefficients by 1/(l(l+1))
// (the adjoint of the analysis, whose fold factors `adjoint` selects).
template <typename T, int CV, int R>
__global__ void __launch_bounds__(32 * kDirWarps, vec_min_ctas<T, CV, R>())
    k_vleg_inv(const T* __restrict__ alm, int nvec, T* __restrict__ F, int64_t Ftot, int Lv, int Mv, int Lp, int Mp,
               Geom geo, const RingLite* __restrict__ rings, const double* __restrict__ z,
               const int* __restrict__ lstart, const double2* __restrict__ pstart,
               const typename DirRec<T>::Coef* __restrict__ coef, const double2* __restrict__ norm, int Lpad,
               const double2* __restrict__ seeds, int csphase, int adjoint, int use_nf) {
    constexpr int NC = 2 * CV, W = kDirWarps, LC = kDirChunk;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_first;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    VecFac<T>* fac = (VecFac<T>*)smem_raw + warp * LC;                      // [W][LC]
    cplx<T>* raw = (cplx<T>*)((VecFac<T>*)smem_raw + W * LC);               // [2][W][LC][NC]: (S, T) per map
    T* rows = (T*)(raw + 2 * W * LC * NC) + (size_t)warp * LC * 8 * CV;     // [W][LC][A0, A1][2 NC]
    const int NP = geo.NP;
    const int m0 = blockIdx.y * W, m = m0 + warp;
    const int pb = blockIdx.x * 32 * R;
    const int b0 = blockIdx.z * CV;
    if (pb + 32 * R <= geo.first_ring(m0)) return;
    const int mend = min(Mv, Lv);  // orders with coefficients
    const int t0 = m < mend ? geo.first_ring(m) : NP;
    const int64_t mo = min(m, Mp - 1);
    const double2* nm = norm + mo * Lpad;
    const auto ord = VecGen<T>::order((int)mo, Mp, Lp, Lpad, NP, coef, norm);

    VecGen<T> gen[R];
    int lmin = kNoDegree, lmax = -1;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int p = pb + 32 * r + lane;
        gen[r].clear();
        if (p >= t0 && p < NP) {
            const int s = gen[r].init(ord, p, z[p], m, Lv, lstart);
            if (s < Lv) {
                gen[r].seed(ord, p, NP, m, seeds, pstart);
                lmin = min(lmin, s);
                lmax = max(lmax, gen[r].last_start(m));
            }
        }
    }
    lmin = __reduce_min_sync(0xffffffffu, lmin);
    lmax = __reduce_max_sync(0xffffffffu, lmax);
    if (threadIdx.x == 0) s_first = kNoDegree;
    __syncthreads();
    if (lane == 0 && lmin < kNoDegree) atomicMin(&s_first, lmin - m);
    __syncthreads();
    const int ibeg = s_first == kNoDegree ? Lv : s_first & ~(LC - 1);

    auto stage = [&](int buf, int i0) {
        cplx<T>* dst = raw + (size_t)buf * W * LC * NC;
        const int j = threadIdx.x & (W - 1), mm = m0 + j;
        const int64_t lm = (int64_t)Lv * Mv;
        for (int k = threadIdx.x / W; k < LC + W - 1; k += 32) {
            const int i = k - j, l = m0 + i0 + k;
            if (i < 0 || i >= LC) continue;
            cplx<T>* d = dst + (j * LC + i) * NC;
            const bool ok = l < Lv && mm < Mv;
            const int64_t o = (int64_t)2 * b0 * lm + (int64_t)l * Mv + mm;
#pragma unroll
            for (int cc = 0; cc < NC; ++cc) {
                if (ok && 2 * b0 + cc < 2 * nvec && HPX_INB(2 * (o + cc * lm) + 1, kExtAlm, 26))
                    cp_async_cplx(d + cc, (const cplx<T>*)alm + o + cc * lm);
                else
                    d[cc] = {(T)0, (T)0};
            }
        }
        cp_async_commit();
    };

    Pair<T> E[R][NC], O[R][NC];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int cc = 0; cc < NC; ++cc) E[r][cc] = O[r][cc] = Pair<T>::zero();
    constexpr int G = 4;  // degrees per unrolled group

    int buf = 0;
    if (m0 + ibeg < Lv) stage(0, ibeg);
    for (int i0 = ibeg; m0 + i0 < Lv; i0 += LC, buf ^= 1) {
        if (m0 + i0 + LC < Lv) {
            stage(buf ^ 1, i0 + LC);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        const int lc = m + i0;
        if (lc < Lv && lmin < lc + LC) {
            // rows of degree lc + lane: A0 = c (S, -T), A1 = c m (i T, i S) as re, im pairs
            const int l = lc + lane;
            fac[lane] = VecFac<T>::make(l, m, nm, Lv);
            double c = sizeof(T) == 4 && l < Lv ? nm[l].x : 1.0;
            if (use_nf && l > 0) c *= 1.0 / ((double)l * (double)(l + 1));
            if (csphase && (m & 1)) c = -c;
            const double cb = VecGen<T>::kScaled ? c * m : c;
            const cplx<T>* sr = raw + ((size_t)(buf * W + warp) * LC + lane) * NC;
            cplx<T>* row = (cplx<T>*)(rows + lane * 8 * CV);
#pragma unroll
            for (int vb = 0; vb < CV; ++vb) {
                const cplx<T> Sv = sr[2 * vb], Tv = sr[2 * vb + 1];
                row[2 * vb] = {(T)(c * Sv.re), (T)(c * Sv.im)};
                row[2 * vb + 1] = {(T)(-c * Tv.re), (T)(-c * Tv.im)};
                row[NC + 2 * vb] = {(T)(-cb * Tv.im), (T)(cb * Tv.re)};
                row[NC + 2 * vb + 1] = {(T)(-cb * Sv.im), (T)(cb * Sv.re)};
            }
            __syncwarp();
            auto group = [&](int k, auto starts) {
                const int lg = lc + k;
#pragma unroll
                for (int i = 0; i < G; ++i) {
                    const auto ab = VecGen<T>::load(ord, lg + i);
                    const VecFac<T> fl = fac[k + i];
                    Pair<T> a0[NC], a1[NC];
                    load_pairs<NC>(a0, rows + (k + i) * 8 * CV);
                    load_pairs<NC>(a1, rows + (k + i) * 8 * CV + 2 * NC);
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        if constexpr (decltype(starts)::value) gen[r].start(ord, pb + 32 * r + lane, lg + i, pstart);
                        T p0, p1;
                        gen[r].value(fl, m, p0, p1);
                        const Pair<T> pp0 = Pair<T>::make(p0, p0), pp1 = Pair<T>::make(p1, p1);
#pragma unroll
                        for (int cc = 0; cc < NC; ++cc) {
                            ((i & 1) ? E[r][cc] : O[r][cc]).fma(pp0, a0[cc]);
                            ((i & 1) ? O[r][cc] : E[r][cc]).fma(pp1, a1[cc]);
                        }
                        gen[r].advance(ab);
                    }
                }
            };
            int k = max(0, lmin - lc) & ~(G - 1);
            const int kend = min(LC, Lv - lc);
            const int ks = min(kend, max(0, lmax - lc + 1));
#pragma unroll 1
            for (; k < ks; k += G) group(k, DirYes{});
#pragma unroll 1
            for (; k < kend; k += G) group(k, DirNo{});
        }
        __syncthreads();
    }
    cplx<T>* Fo = (cplx<T>*)smem_raw;  // [E + O, E - O][column][ring][order]
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int cc = 0; cc < NC; ++cc) {
            const auto e = E[r][cc].get(), o = O[r][cc].get();
            const int k = 32 * r + lane;
            Fo[(cc * 32 * R + k) * W + (warp ^ (k & (W - 1)))] = {e.x + o.x, e.y + o.y};
            Fo[((NC + cc) * 32 * R + k) * W + (warp ^ (k & (W - 1)))] = {e.x - o.x, e.y - o.y};
        }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < R; ++kk) {
        const int j = threadIdx.x & (W - 1), k = kk * 32 + threadIdx.x / W, p = pb + k, mj = m0 + j;
        if (p >= NP) continue;
        const RingLite rl = rings[p];
        if (mj >= rl.mt) continue;
        double s0 = 1.0;
        if (adjoint) s0 = (mj == 0 || mj == rl.h) ? rl.w : 0.5 * rl.w;
        const T sc = (T)(VecGen<T>::kScaled ? s0 * rl.rs : s0);
#pragma unroll
        for (int cc = 0; cc < NC; ++cc) {
            if (2 * b0 + cc >= 2 * nvec) break;
            const int64_t fb = (int64_t)(2 * b0 + cc) * Ftot + mj;
            const int jj = j ^ (k & (W - 1));
            if (HPX_INB(2 * (fb + rl.foff_n) + 1, kExtF, 19))
                ((cplx<T>*)F)[fb + rl.foff_n] = cscale(Fo[(cc * 32 * R + k) * W + jj], sc);
            if (rl.foff_s >= 0 && HPX_INB(2 * (fb + rl.foff_s) + 1, kExtF, 19))
                ((cplx<T>*)F)[fb + rl.foff_s] = cscale(Fo[((NC + cc) * 32 * R + k) * W + jj], sc);
        }
    }
}

}  // namespace hpx
