// Legendre contractions for few columns, straight from and to the ring spectra.
//
// With up to a few maps the contraction has next to nothing to multiply: one
// Pbar value meets 2 real columns per map, while generating it costs two or three
// FP64 operations and (FP32 plans) one FP64 -> FP32 conversion.  So here the work is
// laid out for the generator.  A warp owns one order m and 32 R rings, lane by
// lane: R independent FP64 recurrences per lane keep the FP64 pipe fed without
// any other warp's help, every value is used from the register that produced
// it, and nothing synchronises inside the loop over degrees.
//
//   synthesis  each lane accumulates its rings' even and odd sums in registers
//              and stores the ring spectra F_t = E + O, F_t' = E - O itself;
//   analysis   each lane holds its rings' folded spectra S = w (F_t + F_t'),
//              D = w (F_t - F_t') in registers; per group of degrees the 32
//              partial sums of 32 lanes are transposed and added by 31 exchanges
//              (one per value instead of five), and the warp adds the row to
//              its own shared-memory accumulators.
//
// Neither direction has a fold, unfold or column-layout launch, and neither
// touches the 64-map column layout of the tiled kernels.
//
// What bounds it: one FP64 -> FP32 conversion per value (16 lanes a clock and
// SM; 33% busy in synthesis at C = 8), C/2 packed FP32 FMAs (36%) and two FP64
// operations (15%); what keeps them from more is latency -- 12 to 16 warps an SM fit beside
// the column values.  Measured against the tiled kernels (64 map columns
// whatever the batch) they replaced, analysis + synthesis contraction alone: one
// map at nside 1024, L = M = 2047, FP32 71.3 -> 2.85 ms; 8 maps at nside 256, L
// = M = 511 1370 -> 266 us; 4 maps at nside 128, L = 511, FP64 1412 -> 125 us.
#pragma once

#include "legendre.cuh"

namespace hpx {

// ------------------------------------------------------------ packed accumulators
// A complex column pair as the arithmetic wants it: two FP32 in one 64-bit
// register pair (fma.rn.f32x2: same rounding as two FMAs, half the issue
// slots), or two FP64.
template <typename T>
struct Pair;
template <>
struct Pair<float> {
    unsigned long long v;
    static __device__ __forceinline__ Pair zero() { return {0ull}; }
    static __device__ __forceinline__ Pair make(float a, float b) {
        Pair r;
        asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
        return r;
    }
    __device__ __forceinline__ float2 get() const {
        float2 r;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
        return r;
    }
    // this += p * x
    __device__ __forceinline__ void fma(Pair p, Pair x) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(v) : "l"(p.v), "l"(x.v)); }
};
template <>
struct Pair<double> {
    double a, b;
    static __device__ __forceinline__ Pair zero() { return {0.0, 0.0}; }
    static __device__ __forceinline__ Pair make(double x, double y) { return {x, y}; }
    __device__ __forceinline__ double2 get() const { return make_double2(a, b); }
    __device__ __forceinline__ void fma(Pair p, Pair x) {
        a = ::fma(p.a, x.a, a);
        b = ::fma(p.b, x.b, b);
    }
};

// N consecutive pairs from shared memory, 16 bytes an access
template <int N>
__device__ __forceinline__ void load_pairs(Pair<float> (&a)[N], const float* p) {
    if constexpr (N == 1) {
        const float2 q = *(const float2*)p;
        a[0] = Pair<float>::make(q.x, q.y);
    } else {
#pragma unroll
        for (int i = 0; i < N; i += 2) {
            const float4 q = *(const float4*)(p + 2 * i);
            a[i] = Pair<float>::make(q.x, q.y);
            a[i + 1] = Pair<float>::make(q.z, q.w);
        }
    }
}
template <int N>
__device__ __forceinline__ void load_pairs(Pair<double> (&a)[N], const double* p) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const double2 q = *(const double2*)(p + 2 * i);
        a[i] = Pair<double>::make(q.x, q.y);
    }
}

constexpr int kDirWarps = 4;   // orders per CTA: 4 consecutive FP32 spectra entries fill a 32-byte sector
constexpr int kDirChunk = 32;  // degrees per staged coefficient chunk (synthesis)
constexpr int kNoDegree = 0x3fffffff;

// What the direct kernels need to know about a ring pair (48 bytes; RingPair is
// almost three times that, and its fields would be gathered one sector each)
struct __align__(16) RingLite {
    int64_t foff_n, foff_s;  // spectrum offsets; foff_s < 0: no south ring
    double w;
    int h, mt;
    double rs;  // 1 / sin(theta), 0 at a pole
    double pad;
};

// Recurrence in the form each precision uses.
//   double: Pbar_l = a_l x Pbar_{l-1} - b_l Pbar_{l-2} as everywhere else;
//   float:  Pbar_l = c_l q_l with c_l = b_l c_{l-2}, c_m = c_{m+1} = 1, so that
//           q_l = alpha_l x q_{l-1} - q_{l-2}: two FP64 operations per value
//           instead of three.  c_l (between about 0.1 and 1.13) is applied in FP64 once
//           per degree: to the finished sums (analysis) or to the coefficients
//           (synthesis).  Past l = L - 1 alpha is zero and q only alternates in sign.
template <typename T>
struct DirRec;
template <>
struct DirRec<float> {
    using Coef = double;  // alpha_l
    static __device__ __forceinline__ void advance(double al, double x, double& u0, double& u1) {
        const double v = fma(al * x, u1, -u0);
        u0 = u1;
        u1 = v;
    }
};
template <>
struct DirRec<double> {
    using Coef = double2;  // (a_l, b_l)
    static __device__ __forceinline__ void advance(double2 ab, double x, double& u0, double& u1) {
        const double v = ab.x * x * u1 - ab.y * u0;
        u0 = u1;
        u1 = v;
    }
};

// Tables of the FP32 form for every order: alpha[m * Lpad + l] and norm[m * Lpad
// + l] = (c_l, 1 / c_l), l = m .. L + 1 (alpha and c are zero elsewhere, so a
// recurrence run past l = L - 1 yields zeros).  Thread per order.
__global__ void k_legendre_norm(int M, int L, int Lpad, const double2* __restrict__ coef, double* __restrict__ alpha,
                                double2* __restrict__ norm) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M) return;
    double c2 = 1.0, c1 = 1.0;
    const int64_t o = (int64_t)m * Lpad;
    for (int l = m; l < L; ++l) {
        double c = 1.0, al = 0.0;
        if (l >= m + 2) {
            const double2 ab = coef[o + l];
            c = ab.y * c2;
            al = ab.x * c1 / c;
        }
        alpha[o + l] = al;
        norm[o + l] = make_double2(c, 1.0 / c);
        c2 = c1;
        c1 = c;
    }
}

struct DirYes {
    static constexpr bool value = true;
};
struct DirNo {
    static constexpr bool value = false;
};

// Values the transposed sum takes at once (FP64: half, their registers are twice as wide)
template <typename T>
constexpr int kSumVals = sizeof(T) == 4 ? 32 : 16;

// Which column a lane keeps at column slot 0: slot k of lane i holds column k ^
// sum_perm(i), of C columns (2 per map: re, im)
template <typename T, int C>
__device__ __forceinline__ int sum_perm(int lane) { return (lane / (kSumVals<T> / C)) & (C - 1); }

// v[k G + i] of every lane, k a column slot and i < G = NV / C -> lane j holds the
// sum over lanes of value (column j / G, i = j mod G), j < NV.  At each step a
// lane keeps one half of its values and adds the partner's copy of that half
// (one exchange per value instead of five).  Which half is a matter of the
// lane: with the columns in plain order two selects per exchange (62 of the
// 124 instructions for 32 values, at half the issue rate); in the lane's own
// order (sum_perm) every lane keeps the lower half of the slots in the steps over
// columns, 28 of the 31 exchanges at C = 8.  Measured, plain against lane's own order:
// FP32 analysis of 8 maps at nside 256 180 -> 164 us, of one at nside 1024 1566 ->
// 1514; FP64, 4 maps at nside 128, L = 511 76 -> 69; spin-1 round trip of 4 fields at
// nside 128 147 -> 138.
template <typename T, int NV, int C>
__device__ __forceinline__ T transpose_sum(T (&v)[NV], int lane) {
#pragma unroll
    for (int s = NV / 2; s; s >>= 1) {
        const bool hi = s < NV / C && (lane & s);
#pragma unroll
        for (int i = 0; i < s; ++i) {
            const T keep = hi ? v[i + s] : v[i];
            const T send = hi ? v[i] : v[i + s];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, s);
        }
    }
#pragma unroll
    for (int s = NV; s < 32; s <<= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], s);
    return v[0];
}

// Start of a ring's recurrence: the pair (P_l, P_{l+1}) in the form of T
template <typename T>
__device__ __forceinline__ double2 dir_start(double2 ps, const double2* __restrict__ nm, int l, int L) {
    if constexpr (sizeof(T) == 4) {
        ps.x *= nm[l].y;
        ps.y *= l + 1 < L ? nm[l + 1].y : 0.0;
    }
    return ps;
}

// CTAs per SM the kernels are compiled for: as many as the registers of 2 C R
// column values, R recurrences and the sums leave without spills (one more
// CTA with spills, or one fewer, measured 0-30% slower throughout)
template <typename T, int C, int R>
constexpr int dir_min_ctas() {
    return sizeof(T) == 4 ? (C * R >= 32 ? 3 : 4) : (R >= 4 || C * R >= 16 ? 3 : 4);
}

// ------------------------------------------------------------ analysis
template <typename T, int C, int R>
__host__ __device__ constexpr size_t fwd_direct_xstride() { return (size_t)C * 32 * R + 4; }  // pairs per order
template <typename T, int C, int R>
__host__ __device__ constexpr size_t fwd_direct_smem(int lch) {
    return kDirWarps * (fwd_direct_xstride<T, C, R>() * 2 * sizeof(T) + (size_t)lch * C * sizeof(T));
}

// alm[b][l][m] (+)= sum_p Pbar_l^m(z_p) X[par][p][b] for m = 4 blockIdx.y + warp,
// degrees l = m + blockIdx.x lch .. + lch, maps (C/2) blockIdx.z .. + C/2.
// lch is a multiple of 64 (the chunk starts at a block seed).  The CTA brings
// the spectra of 32 R ring pairs and its four orders (32-byte runs) into shared
// memory, one block ahead; each warp folds its order's into registers and runs its
// degrees.
// blockIdx.x = nch clears the rows' m > l entries (accumulate = 0).
template <typename T, int C, int R>
__global__ void __launch_bounds__(32 * kDirWarps, dir_min_ctas<T, C, R>())
    k_leg_fwd_direct(const T* __restrict__ F, int64_t Ftot, int nmaps, T* __restrict__ alm, int L, int M, Geom geo,
                     const RingLite* __restrict__ rings, const double* __restrict__ z, const int* __restrict__ lstart,
                     const double2* __restrict__ pstart, const typename DirRec<T>::Coef* __restrict__ coef,
                     const double2* __restrict__ norm, int Lpad, const double2* __restrict__ seeds, int lch, int nch,
                     int adjoint, int accumulate) {
    constexpr int NV = kSumVals<T>, G = NV / C;  // degrees per transposed sum
    constexpr int CB = C / 2;  // maps
    constexpr int W = kDirWarps;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int NP = geo.NP;
    const int b0 = blockIdx.z * CB;
    if ((int)blockIdx.x == nch) {
        // m > l: rows l = blockIdx.y, blockIdx.y + gridDim.y, ... below M - 1, the last that
        // has any (walking all L rows this CTA outlasts the sums where M is small:
        // nside 512, L = 1023, M = 1, 16 maps 446 us a call instead of 352)
        for (int l = blockIdx.y; l < min(L, M - 1); l += gridDim.y)
            for (int bb = 0; bb < CB; ++bb) {
                if (b0 + bb >= nmaps) break;
                cplx<T>* row = (cplx<T>*)alm + ((int64_t)(b0 + bb) * L + l) * M;
                for (int m = l + 1 + threadIdx.x; m < M; m += blockDim.x)
                    if (HPX_INB(2 * (((int64_t)(b0 + bb) * L + l) * M + m) + 1, kExtAlm, 20)) row[m] = {(T)0, (T)0};
            }
        return;
    }
    constexpr size_t XS = fwd_direct_xstride<T, C, R>();
    cplx<T>* Xs = (cplx<T>*)smem_raw;  // [W][XS]: [north, south][map][32 R rings]
    T* acc = (T*)(Xs + W * XS) + (size_t)warp * lch * C;
    const int m0 = blockIdx.y * W, m = m0 + warp;
    const int i0 = blockIdx.x * lch, l0 = m + i0;
    if (m0 + i0 >= L) return;
    const bool active = m < M && l0 < L;
    const int n = active ? min(lch, L - l0) : 0;
    const int ng = (n + G - 1) / G;
    for (int i = lane; i < ng * NV; i += 32) acc[i] = (T)0;
    const int t0 = active ? geo.first_ring(m) : NP;
    const int64_t mo = (int64_t)min(m, M - 1);
    const typename DirRec<T>::Coef* cm = coef + mo * Lpad + 2;
    const double2* nm = norm + mo * Lpad;
    const double2* sm = seeds + (mo * seed_blocks(L) + i0 / kSeedBlock) * NP;

    const int perm = sum_perm<T, C>(lane), acc_lane = (lane % G) * C + lane / G;
    // ring spectra of 32 R pairs: thread = (order j, ring k), 4 orders = 32 (64) contiguous bytes
    auto stage = [&](int pb) {
#pragma unroll
        for (int kk = 0; kk < R; ++kk) {
            const int j = threadIdx.x & (W - 1), k = kk * 32 + threadIdx.x / W, p = pb + k, mj = m0 + j;
            cplx<T>* xd = Xs + j * XS + k;
            RingLite rl{};
            if (p < NP) rl = rings[p];
            const bool ok = mj < rl.mt;  // the ring carries this order
#pragma unroll
            for (int bb = 0; bb < CB; ++bb) {
                const int64_t fb = (int64_t)(b0 + bb) * Ftot + mj;
                const bool in = ok && b0 + bb < nmaps;
                if (in && HPX_INB(2 * (fb + rl.foff_n) + 1, kExtF, 21))
                    cp_async_cplx(xd + bb * 32 * R, (const cplx<T>*)F + fb + rl.foff_n);
                else
                    xd[bb * 32 * R] = {(T)0, (T)0};
                if (in && rl.foff_s >= 0 && HPX_INB(2 * (fb + rl.foff_s) + 1, kExtF, 21))
                    cp_async_cplx(xd + (CB + bb) * 32 * R, (const cplx<T>*)F + fb + rl.foff_s);
                else
                    xd[(CB + bb) * 32 * R] = {(T)0, (T)0};
            }
        }
        cp_async_commit();
    };
    const int pfirst = geo.first_ring(m0);
    if (pfirst < NP) stage(pfirst);
    for (int pb = pfirst; pb < NP; pb += 32 * R) {
        int ls[R];
        double x[R], u0[R], u1[R];
        int lmin = kNoDegree, lmax = -1;  // first and last start after l0 (lmin: or any earlier one)
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int p = pb + 32 * r + lane;
            ls[r] = kNoDegree;
            u0[r] = u1[r] = x[r] = 0.0;
            if (p >= t0 && p < NP) {
                const int s = lstart[mo * NP + p];
                x[r] = z[p];
                if (s < l0 + n) {
                    ls[r] = s;
                    if (s <= l0) {
                        const double2 sd = dir_start<T>(sm[p], nm, l0, L);
                        u0[r] = sd.x;
                        u1[r] = sd.y;
                    } else {
                        lmax = max(lmax, s);
                    }
                }
            }
            lmin = min(lmin, ls[r]);
        }
        lmin = __reduce_min_sync(0xffffffffu, lmin);
        lmax = __reduce_max_sync(0xffffffffu, lmax);
        cp_async_wait<0>();
        __syncthreads();
        // S = w (F_t + F_t'), D = w (F_t - F_t'); the equator (no south ring): S = w F_t, D = 0
        Pair<T> S[R][CB], D[R][CB];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int p = min(pb + 32 * r + lane, NP - 1);
            const bool south = rings[p].foff_s >= 0;
            const T w = adjoint ? ((m == 0 || m == rings[p].h) ? (T)1 : (T)2) : (T)rings[p].w;
#pragma unroll
            for (int bb = 0; bb < CB; ++bb) {
                const cplx<T>* xs = Xs + warp * XS + 32 * r + lane + (bb ^ (perm >> 1)) * 32 * R;
                const cplx<T> a = xs[0], c = xs[CB * 32 * R];
                const cplx<T> sv = cscale(cadd(a, c), w), dv = cscale(csub(a, c), south ? w : (T)0);
                S[r][bb] = perm & 1 ? Pair<T>::make(sv.im, sv.re) : Pair<T>::make(sv.re, sv.im);
                D[r][bb] = perm & 1 ? Pair<T>::make(dv.im, dv.re) : Pair<T>::make(dv.re, dv.im);
            }
        }
        __syncthreads();  // every warp has its rings: the next block's spectra land while this one is used
        if (pb + 32 * R < NP) stage(pb + 32 * R);
        if (lmin == kNoDegree) continue;  // every value of these rings and degrees is below 2^-1000
        int g = max(0, lmin - l0) / G;
        constexpr bool AHEAD = sizeof(T) == 4 && C > 2;  // a group's coefficients one group ahead, if registers allow
        typename DirRec<T>::Coef cn[G];
#pragma unroll
        for (int i = 0; i < (AHEAD ? G : 0); ++i) cn[i] = cm[l0 + g * G + i];
        // G degrees from lg on; STARTS: some ring's recurrence starts among them
        auto group = [&](int g, auto starts) {
            const int lg = l0 + g * G;
            Pair<T> v[G][CB];
#pragma unroll
            for (int i = 0; i < G; ++i)
#pragma unroll
                for (int bb = 0; bb < CB; ++bb) v[i][bb] = Pair<T>::zero();
#pragma unroll
            for (int i = 0; i < G; ++i) {
                const auto ab = AHEAD ? cn[i] : cm[lg + i];
                if constexpr (AHEAD) cn[i] = cm[lg + G + i];
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    if constexpr (decltype(starts)::value) {
                        if (ls[r] == lg + i && ls[r] > l0) {
                            const double2 ps = dir_start<T>(pstart[mo * NP + pb + 32 * r + lane], nm, lg + i, L);
                            u0[r] = ps.x;
                            u1[r] = ps.y;
                        }
                    }
                    const T pv = (T)u0[r];
                    const Pair<T> pp = Pair<T>::make(pv, pv);
#pragma unroll
                    for (int bb = 0; bb < CB; ++bb) v[i][bb].fma(pp, (i & 1) ? D[r][bb] : S[r][bb]);
                    DirRec<T>::advance(ab, x[r], u0[r], u1[r]);
                }
            }
            T f[NV];
#pragma unroll
            for (int i = 0; i < G; ++i)
#pragma unroll
                for (int bb = 0; bb < CB; ++bb) {
                    const auto q = v[i][bb].get();
                    f[2 * bb * G + i] = q.x;
                    f[(2 * bb + 1) * G + i] = q.y;
                }
            const T sum = transpose_sum<T, NV, C>(f, lane);  // lane = column G + degree in group
            if (lane < NV) acc[g * NV + acc_lane] += sum;
        };
        const int gs = lmax < 0 ? g : min(ng, (lmax - l0) / G + 1);  // later groups start no ring
#pragma unroll 1
        for (; g < gs; ++g) group(g, DirYes{});
#pragma unroll 1
        for (; g < ng; ++g) group(g, DirNo{});
    }
    __syncwarp();
    for (int i = lane; i < n; i += 32) {
        const double c = sizeof(T) == 4 ? nm[l0 + i].x : 1.0;
#pragma unroll
        for (int bb = 0; bb < CB; ++bb) {
            if (b0 + bb >= nmaps) break;
            const int64_t o = ((int64_t)(b0 + bb) * L + l0 + i) * M + m;
            if (!HPX_INB(2 * o + 1, kExtAlm, 22)) continue;
            cplx<T> q = *(const cplx<T>*)(acc + i * C + 2 * bb);
            if constexpr (sizeof(T) == 4) q = {(T)((double)q.re * c), (T)((double)q.im * c)};
            cplx<T>* dst = (cplx<T>*)alm + o;
            if (accumulate) q = cadd(*dst, q);
            *dst = q;
        }
    }
}

// ------------------------------------------------------------ synthesis
// shared memory: two coefficient chunks, reused for the outgoing spectra
template <typename T, int C, int R>
__host__ __device__ constexpr size_t inv_direct_smem() {
    const size_t a = (size_t)2 * kDirWarps * kDirChunk * C * sizeof(T);
    const size_t f = (size_t)2 * kDirWarps * 32 * R * C * sizeof(T);
    return a > f ? a : f;
}

// F[b][foff_t + m] = sc (E + O), F[b][foff_t' + m] = sc (E - O) for orders
// m = 4 blockIdx.y + warp, rings 32 R blockIdx.x .. + 32 R, maps (C/2) blockIdx.z
// .. + C/2; sc = 1, or for the adjoint of analysis w_t (m = 0, nphi/2) and w_t/2.
// The CTA's warps walk the degrees together, 32 at a time counted from each
// warp's own m; their coefficients (4 consecutive orders: 32-byte runs of every
// row) are double-buffered through shared memory by cp.async, and the spectra
// leave through shared memory in the same runs.
template <typename T, int C, int R>
__global__ void __launch_bounds__(32 * kDirWarps, dir_min_ctas<T, C, R>())
    k_leg_inv_direct(const T* __restrict__ alm, int nmaps, T* __restrict__ F, int64_t Ftot, int L, int M, Geom geo,
                     const RingLite* __restrict__ rings, const double* __restrict__ z, const int* __restrict__ lstart,
                     const double2* __restrict__ pstart, const typename DirRec<T>::Coef* __restrict__ coef,
                     const double2* __restrict__ norm, int Lpad, int adjoint) {
    constexpr int CB = C / 2, W = kDirWarps, LC = kDirChunk;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_first;
    T* As = (T*)smem_raw;  // [2][W][LC][C]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int NP = geo.NP;
    const int m0 = blockIdx.y * W, m = m0 + warp;
    const int pb = blockIdx.x * 32 * R;
    const int b0 = blockIdx.z * CB;
    if (pb + 32 * R <= geo.first_ring(m0)) return;  // no order of this CTA reaches these rings
    const int t0 = m < M ? geo.first_ring(m) : NP;
    const int64_t mo = min(m, M - 1);
    const typename DirRec<T>::Coef* cm = coef + mo * Lpad + 2;
    const double2* nm = norm + mo * Lpad;

    int ls[R];
    double x[R], u0[R], u1[R];
    int lmin = kNoDegree, lmax = -1;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int p = pb + 32 * r + lane;
        ls[r] = kNoDegree;
        x[r] = u0[r] = u1[r] = 0.0;
        if (p >= t0 && p < NP && m < L) {
            const int s = lstart[mo * NP + p];
            x[r] = z[p];
            if (s < L) {
                ls[r] = s;
                lmax = max(lmax, s);
            }
        }
        lmin = min(lmin, ls[r]);
    }
    lmin = __reduce_min_sync(0xffffffffu, lmin);
    lmax = __reduce_max_sync(0xffffffffu, lmax);
    if (threadIdx.x == 0) s_first = kNoDegree;
    __syncthreads();
    if (lane == 0 && lmin < kNoDegree) atomicMin(&s_first, lmin - m);
    __syncthreads();
    const int ibeg = s_first == kNoDegree ? L : s_first & ~(LC - 1);

    // degrees m + i0 .. m + i0 + LC of every order of the CTA: row l = m0 + i0 + k
    // holds order m0 + j at its own offset k - j
    auto stage = [&](int buf, int i0) {
        T* dst = As + (size_t)buf * W * LC * C;
        const int j = threadIdx.x & (W - 1), mm = m0 + j;
        const int64_t lm = (int64_t)L * M;
        for (int k = threadIdx.x / W; k < LC + W - 1; k += 32) {
            const int i = k - j, l = m0 + i0 + k;
            if (i < 0 || i >= LC) continue;
            cplx<T>* d = (cplx<T>*)(dst + (j * LC + i) * C);
            const bool ok = l < L && mm < M;
            const int64_t o = (int64_t)b0 * lm + (int64_t)l * M + mm;
#pragma unroll
            for (int bb = 0; bb < CB; ++bb) {
                if (ok && b0 + bb < nmaps && HPX_INB(2 * (o + bb * lm) + 1, kExtAlm, 23))
                    cp_async_cplx(d + bb, (const cplx<T>*)alm + o + bb * lm);
                else
                    d[bb] = {(T)0, (T)0};
            }
        }
        cp_async_commit();
    };

    Pair<T> E[R][CB], O[R][CB];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int bb = 0; bb < CB; ++bb) E[r][bb] = O[r][bb] = Pair<T>::zero();
    constexpr int G = sizeof(T) == 4 ? 8 : 4;  // degrees per unrolled group

    int buf = 0;
    if (m0 + ibeg < L) stage(0, ibeg);
    for (int i0 = ibeg; m0 + i0 < L; i0 += LC, buf ^= 1) {
        if (m0 + i0 + LC < L) {
            stage(buf ^ 1, i0 + LC);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        T* aw = As + (size_t)(buf * W + warp) * LC * C;
        const int lc = m + i0;
        if (lc < L && lmin < lc + LC) {
            if constexpr (sizeof(T) == 4) {
                // a_l c_l (the recurrence carries Pbar_l / c_l); C lanes share a degree's norm
#pragma unroll
                for (int q = 0; q < LC * C / 2; q += 32) {
                    cplx<T>* e = (cplx<T>*)aw + q + lane;
                    const int l = lc + (q + lane) / CB;
                    const double c = l < L ? nm[l].x : 0.0;
                    const cplx<T> v = *e;
                    *e = {(T)((double)v.re * c), (T)((double)v.im * c)};
                }
                __syncwarp();
            }
            int k = max(0, lmin - lc) & ~(G - 1);
            constexpr bool AHEAD = sizeof(T) == 4;  // a group's coefficients one group ahead, if registers allow
            typename DirRec<T>::Coef cn[G];
#pragma unroll
            for (int i = 0; i < (AHEAD ? G : 0); ++i) cn[i] = cm[lc + k + i];
            auto group = [&](int k, auto starts) {
                const int lg = lc + k;
#pragma unroll
                for (int i = 0; i < G; ++i) {
                    const auto ab = AHEAD ? cn[i] : cm[lg + i];
                    if constexpr (AHEAD) cn[i] = cm[lg + G + i];
                    Pair<T> a[CB];
                    load_pairs<CB>(a, aw + (k + i) * C);
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        if constexpr (decltype(starts)::value) {
                            if (ls[r] == lg + i) {
                                const double2 ps = dir_start<T>(pstart[mo * NP + pb + 32 * r + lane], nm, lg + i, L);
                                u0[r] = ps.x;
                                u1[r] = ps.y;
                            }
                        }
                        const T pv = (T)u0[r];
                        const Pair<T> pp = Pair<T>::make(pv, pv);
#pragma unroll
                        for (int bb = 0; bb < CB; ++bb) ((i & 1) ? O[r][bb] : E[r][bb]).fma(pp, a[bb]);
                        DirRec<T>::advance(ab, x[r], u0[r], u1[r]);
                    }
                }
            };
            const int kend = min(LC, L - lc);
            const int ks = min(kend, max(0, lmax - lc + 1));  // later groups start no ring
#pragma unroll 1
            for (; k < ks; k += G) group(k, DirYes{});
#pragma unroll 1
            for (; k < kend; k += G) group(k, DirNo{});
        }
        __syncthreads();  // the buffer is restaged in the next iteration
    }
    // E + O and E - O to shared memory [pol][map][ring][order], then 4 orders at a time to F
    cplx<T>* Fo = (cplx<T>*)smem_raw;
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int bb = 0; bb < CB; ++bb) {
            const auto e = E[r][bb].get(), o = O[r][bb].get();
            const int k = 32 * r + lane;
            Fo[(bb * 32 * R + k) * W + (warp ^ (k & (W - 1)))] = {e.x + o.x, e.y + o.y};
            Fo[((CB + bb) * 32 * R + k) * W + (warp ^ (k & (W - 1)))] = {e.x - o.x, e.y - o.y};
        }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < R; ++kk) {
        const int j = threadIdx.x & (W - 1), k = kk * 32 + threadIdx.x / W, p = pb + k, mj = m0 + j;
        if (p >= NP) continue;
        const RingLite rl = rings[p];
        if (mj >= rl.mt) continue;
        T sc = (T)1;
        if (adjoint) sc = (mj == 0 || mj == rl.h) ? (T)rl.w : (T)(0.5 * rl.w);
#pragma unroll
        for (int bb = 0; bb < CB; ++bb) {
            if (b0 + bb >= nmaps) break;
            const int64_t fb = (int64_t)(b0 + bb) * Ftot + mj;
            const int jj = j ^ (k & (W - 1));
            if (HPX_INB(2 * (fb + rl.foff_n) + 1, kExtF, 24))
                ((cplx<T>*)F)[fb + rl.foff_n] = cscale(Fo[(bb * 32 * R + k) * W + jj], sc);
            if (rl.foff_s >= 0 && HPX_INB(2 * (fb + rl.foff_s) + 1, kExtF, 24))
                ((cplx<T>*)F)[fb + rl.foff_s] = cscale(Fo[((CB + bb) * 32 * R + k) * W + jj], sc);
        }
    }
}

}  // namespace hpx
