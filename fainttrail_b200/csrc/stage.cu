// The time-order-dependent preprocessing stage on the B200: FaintTrail's
// build_stage (preprocess.cpp:286-486) for a whole image with a fixed PSF width,
// bit-identical to the reference CPU code.
//
//  sky_middle_kernel, sky_kernel (more than 128 frames)
//                  static sky + leave-out residuals (preprocess.cpp:154-204)
//  sample + select per-frame residual noise: regular sample grid, exact medians
//                  by bracketing and radix selection (common.hpp:64-100, preprocess.cpp:356-365)
//  scatter_net_kernel, scatter_kernel (more than 128 frames)
//                  temporal scatter (preprocess.cpp:373-391)
//  mask_kernel     dilated scatter mask (preprocess.cpp:392-400)
//  filter_frames_kernel, filter_kernel (wide PSFs)
//                  normalise + weight, cosmic-ray rejection, clip, separable
//                  matched filter, fused per tile (preprocess.cpp:414-451, 116-148)
//  sample + select robust sigma of the filter output, then rescale
//                  (preprocess.cpp:454-471)
//
// Arithmetic follows the reference operation by operation: float adds and
// multiplies with round-to-nearest and no contraction, double where the
// reference promotes to double, the same summation orders, NaN rules and casts.
#include <cooperative_groups.h>
#include <math_constants.h>

#include <algorithm>
#include <cmath>
#include <numeric>
#include <type_traits>
#include <vector>

#include "engine.h"
#include "search.h"
#include "stage.h"

namespace ftb {

namespace {

namespace cg = cooperative_groups;

constexpr double kFwhmToSigma = 1.0 / 2.354820045030949;  // psf.hpp:16

__device__ __forceinline__ bool finitef(float v) { return isfinite(v); }

// ------------------------------------------------------------------ static sky

struct SkyArgs {
    const float* sub;
    float* residual;
    float* sky;
    const unsigned char* frame_of;  // frame of each time rank
    int w, h, pitch, n, exclude, need;
    int sub_pitch;  // of sub, any
};

// One thread per pixel. The pixel's values are held in time-rank order, so the
// reference's sort of (value, time rank) pairs orders equal values by index.
// Each finite value's sorted position is counted against all others, eight
// values per pass over the column (the non-finite ones are held as +inf and
// never counted). The leave-out median of the frame of rank r is then the lo-th /
// hi-th sorted value outside the exclusion window [r - exclude, r + exclude]; the
// window's sorted positions are a bitmask that slides one rank per
// frame (one position leaves, one enters), and the kept positions are picked
// with popc / fns.
// flips sorted position p (255: a non-finite value, no position) in the window
// mask; returns 1 if a position was flipped
constexpr int kSkyWords = 8;  // 256 sorted positions
__device__ __forceinline__ int sky_toggle(uint32_t (&ex)[kSkyWords], int p) {
    if (p == 255) return 0;
#pragma unroll
    for (int wd = 0; wd < kSkyWords; ++wd) ex[wd] ^= (p >> 5) == wd ? 1u << (p & 31) : 0u;
    return 1;
}

// Position of the k-th (0-based) set bit of x, k < popc(x): a binary search on
// the population counts of halves.
__device__ __forceinline__ int nth_set_bit(uint32_t x, int k) {
    int pos = 0;
    int c = __popc(x & 0xffffu);
    if (k >= c) { k -= c; pos += 16; x >>= 16; }
    c = __popc(x & 0xffu);
    if (k >= c) { k -= c; pos += 8; x >>= 8; }
    c = __popc(x & 0xfu);
    if (k >= c) { k -= c; pos += 4; x >>= 4; }
    c = __popc(x & 0x3u);
    if (k >= c) { k -= c; pos += 2; x >>= 2; }
    if (k >= static_cast<int>(x & 1u)) pos += 1;
    return pos;
}

// The static sky and the leave-out residuals of one pixel from its values by
// time rank (V, +inf where not finite), its m_all finite values in sorted order
// (S) and each rank's sorted position (PF, 255 where not finite).
__device__ __forceinline__ void sky_finish(const SkyArgs& a, const float* V, const float* S, const unsigned char* PF,
                                           int T, int t, int m_all, size_t pix, size_t plane) {
    const int n = a.n;
    // global median: the two middle floats are added in float (preprocess.cpp:171)
    const float mid_sum = __fadd_rn(S[((m_all - 1) / 2) * T + t], S[(m_all / 2) * T + t]);
    const double global = 0.5 * static_cast<double>(mid_sum);
    a.sky[pix] = __double2float_rn(global);
    uint32_t ex[kSkyWords];
#pragma unroll
    for (int wd = 0; wd < kSkyWords; ++wd) ex[wd] = 0;
    int excluded = 0;
    if (a.exclude > 0)
        for (int r = 0; r <= min(a.exclude, n - 1); ++r) excluded += sky_toggle(ex, PF[r * T + t]);  // rank 0's window
    for (int r = 0; r < n; ++r) {
        if (a.exclude > 0 && r > 0) {
            if (r - 1 - a.exclude >= 0) excluded -= sky_toggle(ex, PF[(r - 1 - a.exclude) * T + t]);
            if (r + a.exclude < n) excluded += sky_toggle(ex, PF[(r + a.exclude) * T + t]);
        }
        const float v = V[r * T + t];
        float* out = a.residual + a.frame_of[r] * plane + pix;
        if (v == CUDART_INF_F) {
            *out = CUDART_NAN_F;
            continue;
        }
        double st = global;
        const int m = m_all - excluded;
        if (a.exclude > 0 && m >= 5) {
            const int lo = (m - 1) / 2, hi = m / 2;
            int plo = -1, phi = -1, seen = 0;
#pragma unroll
            for (int wd = 0; wd < kSkyWords; ++wd) {
                const int nb = min(32, max(0, m_all - wd * 32));
                const uint32_t valid = nb >= 32 ? 0xffffffffu : ((1u << nb) - 1u);
                const uint32_t keep = ~ex[wd] & valid;
                const int c = __popc(keep);
                if (plo < 0 && lo < seen + c) plo = wd * 32 + nth_set_bit(keep, lo - seen);
                if (phi < 0 && hi < seen + c) phi = wd * 32 + nth_set_bit(keep, hi - seen);
                seen += c;
            }
            // double add of the two middle values (preprocess.cpp:198)
            st = 0.5 * (static_cast<double>(S[plo * T + t]) + static_cast<double>(S[phi * T + t]));
        }
        *out = __double2float_rn(static_cast<double>(v) - st);
    }
}

__global__ void __launch_bounds__(64) sky_kernel(const SkyArgs a) {
    extern __shared__ unsigned char sm[];
    const int T = blockDim.x, t = threadIdx.x;
    const int n = a.n;
    float* V = reinterpret_cast<float*>(sm);                            // [n][T] values by time rank, +inf if not finite
    float* S = V + n * T;                                               // [n][T] finite values in sorted order
    unsigned char* PF = reinterpret_cast<unsigned char*>(S + n * T);    // [n][T] sorted position by rank, 255: none
    const long long q = static_cast<long long>(blockIdx.x) * T + t;
    const int x = static_cast<int>(q % a.w), y = static_cast<int>(q / a.w);
    if (y >= a.h) return;
    const size_t plane = static_cast<size_t>(a.pitch) * a.h;
    const size_t pix = static_cast<size_t>(y) * a.pitch + x;
    int m_all = 0;
    for (int r = 0; r < n; ++r) {
        const float v = a.sub[a.frame_of[r] * (static_cast<size_t>(a.sub_pitch) * a.h) + static_cast<size_t>(y) * a.sub_pitch + x];
        const bool fin = finitef(v);
        V[r * T + t] = fin ? v : CUDART_INF_F;
        m_all += fin;
    }
    if (m_all < a.need) {
        a.sky[pix] = CUDART_NAN_F;
        for (int i = 0; i < n; ++i) a.residual[i * plane + pix] = CUDART_NAN_F;
        return;
    }
    constexpr int B = 8;
    for (int e0 = 0; e0 < n; e0 += B) {
        float ve[B];
        int pos[B];
#pragma unroll
        for (int b = 0; b < B; ++b) {
            ve[b] = e0 + b < n ? V[(e0 + b) * T + t] : CUDART_INF_F;
            pos[b] = 0;
        }
        for (int f = 0; f < e0; ++f) {  // lower ranks: equal values sort first
            const float vf = V[f * T + t];
#pragma unroll
            for (int b = 0; b < B; ++b) pos[b] += vf <= ve[b];
        }
        const int e1 = min(e0 + B, n);
        if (e1 - e0 == B) {
            // a full block against itself: rank e0 + c before rank e0 + b sorts an
            // equal value first, so the comparison is fixed per (c, b) pair
#pragma unroll
            for (int c = 0; c < B; ++c) {
                const float vf = V[(e0 + c) * T + t];
#pragma unroll
                for (int b = 0; b < B; ++b) pos[b] += c < b ? vf <= ve[b] : vf < ve[b];
            }
        } else {
            for (int f = e0; f < e1; ++f) {
                const float vf = V[f * T + t];
#pragma unroll
                for (int b = 0; b < B; ++b) pos[b] += vf < ve[b] || (vf == ve[b] && f < e0 + b);
            }
        }
        for (int f = e1; f < n; ++f) {  // higher ranks: only smaller values
            const float vf = V[f * T + t];
#pragma unroll
            for (int b = 0; b < B; ++b) pos[b] += vf < ve[b];
        }
#pragma unroll
        for (int b = 0; b < B; ++b) {
            if (e0 + b >= n) break;
            const bool fin = ve[b] != CUDART_INF_F;
            if (fin) S[pos[b] * T + t] = ve[b];
            PF[(e0 + b) * T + t] = fin ? static_cast<unsigned char>(pos[b]) : 255;
        }
    }
    sky_finish(a, V, S, PF, T, t, m_all, pix, plane);
}

// ---- the same for n <= N <= 128, without sorted positions for all values
//
// Leaving out x of the m sorted values moves the median's position by at most x, so
// with windows of at most X ranks every median lies at the sorted positions [(m - X -
// 1) / 2, (m + X) / 2], about a quarter of them at the default window. The values are
// sorted by a network in registers (Batcher's merge exchange), those middle ones kept
// in shared memory, and a window's content is the number of its values below them and
// a bitmask of the middle positions it takes. Equal values are interchangeable: one
// that enters takes the first free position from its run's first on, one that leaves
// frees the run's first taken one; where a run reaches beyond the middle, its
// count says which part the next one belongs to. Only the two zeros are equal and
// differ, which shows in the sky alone (a residual against one or the other differs at
// most in the sign of a zero, which no sum, product or comparison after it sees): where
// the pixel holds a -0.0 and its median is zero, the wanted one is looked up in rank
// order.
//
// Bound by issue, mostly of the integer and compare pipe: 173 instructions a value at
// 40 frames (a third of them in the loop over the ranks) where counting every rank
// against all others and finishing on full masks took 330. 40 frames of 2048^2: 1.71
// -> 1.01 ms; 120 of 1030 x 777 (a bitonic network, 64 threads a CTA with all
// positions in shared memory): 5.46 -> 1.35 ms; 33 of 1501 x 1117: 0.57 -> 0.35 ms.
// Whole numbers with a standard deviation of 33, most of whose pixels have equal values at
// the middle's ends: 1.71 -> 1.45 and 7.59 -> 2.78 ms.

// Masks: position of the lowest set bit (x != 0), of the k-th (0-based) set bit (k <
// popc(x), x below 2^16 where small), and bit c, or 0 for a c beyond the mask.
__device__ __forceinline__ int low_bit(uint32_t x) { return __ffs(static_cast<int>(x)) - 1; }
__device__ __forceinline__ int low_bit(uint64_t x) { return __ffsll(static_cast<long long>(x)) - 1; }
__device__ __forceinline__ int low_bit(unsigned __int128 x) {
    const uint64_t lo = static_cast<uint64_t>(x);
    return lo ? low_bit(lo) : 64 + low_bit(static_cast<uint64_t>(x >> 64));
}
__device__ __forceinline__ int nth_bit(uint32_t x, int k, bool small) {
    int pos = 0;
    if (!small) {
        const int c = __popc(x & 0xffffu);
        if (k >= c) { k -= c; pos = 16; x >>= 16; }
    }
    int c = __popc(x & 0xffu);
    if (k >= c) { k -= c; pos += 8; x >>= 8; }
    c = __popc(x & 0xfu);
    if (k >= c) { k -= c; pos += 4; x >>= 4; }
    c = __popc(x & 0x3u);
    if (k >= c) { k -= c; pos += 2; x >>= 2; }
    return pos + (k >= static_cast<int>(x & 1u));
}
__device__ __forceinline__ int nth_bit(uint64_t x, int k, bool) {
    const uint32_t lo = static_cast<uint32_t>(x);
    const int c = __popc(lo);
    const bool up = k >= c;
    return (up ? 32 : 0) + nth_bit(up ? static_cast<uint32_t>(x >> 32) : lo, up ? k - c : k, false);
}
__device__ __forceinline__ int nth_bit(unsigned __int128 x, int k, bool) {
    const uint64_t lo = static_cast<uint64_t>(x);
    const int c = __popcll(lo);
    const bool up = k >= c;
    return (up ? 64 : 0) + nth_bit(up ? static_cast<uint64_t>(x >> 64) : lo, up ? k - c : k, false);
}
__device__ __forceinline__ void one_bit(uint32_t& x, unsigned c) { asm("shl.b32 %0, 1, %1;" : "=r"(x) : "r"(c)); }
__device__ __forceinline__ void one_bit(uint64_t& x, unsigned c) { asm("shl.b64 %0, 1, %1;" : "=l"(x) : "r"(c)); }
__device__ __forceinline__ void one_bit(unsigned __int128& x, unsigned c) {
    x = c < 128u ? static_cast<unsigned __int128>(1) << c : 0;
}

// A rank's code: in its low bits its run's first middle position, or none (the masks'
// one_bit gives 0), or a run that reaches beyond the middle (equal to its first value;
// to its last, and not the first); above them, signed, what its exclusion adds to u =
// kept values - 2 (kept values below the middle): 0 for a non-finite value, 1 below the
// middle, else -1. The median's lower position is the (u - 1) / 2-th kept one of the
// middle.
template <class Mask>
struct SkyCode {
    using type = short;
    static constexpr int bits = 9;
};
template <>
struct SkyCode<uint32_t> {
    using type = signed char;
    static constexpr int bits = 6;
};

__host__ __device__ constexpr int sky_threads(int N) { return N <= 64 ? 128 : 64; }
// Positions of the middle at most, for a window of 2 exclude + 1 ranks, and the rows
// that a halving search over them reads (2^k - 1).
__host__ __device__ inline int sky_middle(int n, int exclude) {
    const int x = exclude < n ? 2 * exclude + 1 : n;
    return x + 2 < n ? x + 2 : n;
}
__host__ __device__ inline int sky_rows(int middle) {
    int r = 1;
    while (r < middle) r = 2 * r + 1;
    return r;
}

template <int N, class Mask>
__global__ void __launch_bounds__(sky_threads(N)) sky_middle_kernel(const SkyArgs a) {
    extern __shared__ __align__(16) unsigned char sm[];
    using Code = typename SkyCode<Mask>::type;
    constexpr int T = sky_threads(N), kBits = SkyCode<Mask>::bits;
    constexpr int kNone = (1 << kBits) - 1, kFirst = kNone - 1, kLast = kNone - 2;
    constexpr int kBelow = 1 << kBits, kOther = -(1 << kBits);
    // frames that are there for certain: launch_sky takes the smallest network
    constexpr int kSure = sizeof(Mask) > 4 ? 0 : N <= 64 ? N - 8 : N - 16;
    constexpr bool kHeld = N <= 64;  // the values stay in shared memory; more are read again
    const int t = threadIdx.x, n = a.n, e = min(a.exclude, n), most = sky_middle(n, e), rows = sky_rows(most);
    size_t* at = reinterpret_cast<size_t*>(sm);           // [n] a rank's frame in the residuals, from the first pixel
    size_t* from = at + n;                                // [n] and in sub
    float* S = reinterpret_cast<float*>(from + n) + t;    // [rows][T] the middle values, then +inf
    float* V = S + rows * T;                          // [n][T] values by time rank, +inf if not finite
    // [n + 2 e + 1][T] by time rank, from rank -e - 1 on: none outside the sequence
    Code* code = reinterpret_cast<Code*>(S - t + T * (rows + (kHeld ? n : 0))) + t + T * (e + 1);
    const size_t plane = static_cast<size_t>(a.pitch) * a.h;
    for (int r = t; r < n; r += T) {
        at[r] = a.frame_of[r] * plane;
        from[r] = a.frame_of[r] * (static_cast<size_t>(a.sub_pitch) * a.h);
    }
    __syncthreads();
    const unsigned q = blockIdx.x * static_cast<unsigned>(T) + t;
    const int y = static_cast<int>(q / static_cast<unsigned>(a.w)), x = static_cast<int>(q - y * static_cast<unsigned>(a.w));
    if (y >= a.h) return;
    const size_t pix = static_cast<size_t>(y) * a.pitch + x;
    const float* sub = a.sub + static_cast<size_t>(y) * a.sub_pitch + x;
    float* residual = a.residual + pix;
    float sv[N];
#pragma unroll
    for (int r = 0; r < N; ++r) sv[r] = r < kSure || r < n ? __ldg(sub + from[r]) : CUDART_INF_F;
    int m_all = 0;
    bool negzero = false;
#pragma unroll
    for (int r = 0; r < N; ++r) {
        if (!finitef(sv[r])) sv[r] = CUDART_INF_F;
        m_all += sv[r] != CUDART_INF_F;
        negzero |= __float_as_uint(sv[r]) == 0x80000000u;
        if (kHeld && (r < kSure || r < n)) V[r * T] = sv[r];
    }
    if (m_all < a.need) {
        a.sky[pix] = CUDART_NAN_F;
        for (int i = 0; i < n; ++i) residual[i * plane] = CUDART_NAN_F;
        return;
    }
    auto value = [&](int r) {
        if (kHeld) return V[r * T];
        const float v = sub[from[r]];
        return finitef(v) ? v : CUDART_INF_F;
    };
#pragma unroll
    for (int p = 1; p < N; p <<= 1)
#pragma unroll
        for (int k = p; k > 0; k >>= 1)
#pragma unroll
            for (int i = 0; i < N; ++i)
                if (i >= k % p && i + k < N && ((i - k % p) / k) % 2 == 0 && i / (2 * p) == (i + k) / (2 * p)) {
                    const float lo = fminf(sv[i], sv[i + k]), hi = fmaxf(sv[i], sv[i + k]);
                    sv[i] = lo;
                    sv[i + k] = hi;
                }
    // the middle: positions [first, first + len)
    const int X = e < n ? min(2 * e + 1, n) : n;
    const int first = max(0, (m_all - X - 1) >> 1), len = min(m_all - 1, (m_all + X) >> 1) - first + 1;
    {
        float* to = S - first * T;
#pragma unroll
        for (int p = 0; p < N; ++p)
            if (p >= first && p < first + len) to[p * T] = sv[p];
        for (int p = len; p < rows; ++p) S[p * T] = CUDART_INF_F;
    }
    // the k-th value (0-based) in (value, time rank) order; a zero is looked up, as its sign
    // depends on the order
    auto sorted = [&](int k) {
        float z = S[(k - first) * T];
        if (!negzero || z != 0.0f) return z;
        for (int i = 0; i < n; ++i) k -= value(i) < 0.0f;
        for (int i = 0; i < n && k >= 0; ++i)
            if (value(i) == 0.0f) {
                z = value(i);
                --k;
            }
        return z;
    };
    // global median: the two middle floats are added in float (preprocess.cpp:171)
    const double global = 0.5 * static_cast<double>(__fadd_rn(sorted((m_all - 1) / 2), sorted(m_all / 2)));
    a.sky[pix] = __double2float_rn(global);
    if (e <= 0) {
        for (int r = 0; r < n; ++r) {
            const float v = value(r);
            residual[at[r]] = v != CUDART_INF_F ? __double2float_rn(static_cast<double>(v) - global) : CUDART_NAN_F;
        }
        return;
    }
    auto lower_bound = [&](float v) {
        int p = 0;
#pragma unroll
        for (int s = 4 * static_cast<int>(sizeof(Mask)); s > 0; s >>= 1)
            if (s < rows + 1 && S[(p + s - 1) * T] < v) p += s;
        return p;
    };
    // runs that reach beyond the middle's ends: values of the first below it, and where
    // the last one's starts
    int run_below, run_last = 0;
    bool runs;
    {
        const float s0 = S[0], s1 = S[(len - 1) * T];
        int less = 0, upto = 0;  // values below the first, up to the last
#pragma unroll 4
        for (int r = 0; r < n; ++r) {
            const float v = value(r);
            const int p = lower_bound(v);
            const bool below = v < s0;
            less += below;
            upto += v <= s1;
            const int c = below ? kNone + kBelow : v <= s1 ? p + kOther : v != CUDART_INF_F ? kNone + kOther : kNone;
            code[r * T] = static_cast<Code>(c);
        }
        run_below = first - less;
        const bool beyond = upto > first + len;
        runs = run_below > 0 || beyond;
        if (runs) {
            run_last = lower_bound(s1);
            for (int r = 0; r < n; ++r) {
                const float v = value(r);
                if (v == s0 && (run_below > 0 || s0 == s1))
                    code[r * T] = static_cast<Code>(kFirst + kOther);
                else if (v == s1 && beyond)
                    code[r * T] = static_cast<Code>(kLast + kOther);
            }
        }
    }
    for (int r = 1; r <= e + 1; ++r) code[-r * T] = static_cast<Code>(kNone);
    for (int r = n; r < n + e; ++r) code[r * T] = static_cast<Code>(kNone);
    Mask out = 0;                     // middle positions in the window
    int u = m_all - 2 * first;        // kept values - 2 (kept ones below the middle)
    int first_out = 0, last_out = 0;  // excluded ones of the runs beyond the middle's ends
    const Mask all = len >= static_cast<int>(8 * sizeof(Mask)) ? ~static_cast<Mask>(0) : (static_cast<Mask>(1) << len) - 1;
    // the position that such a run's next excluded (d = 1) or included (-1) value takes
    auto in_run = [&](int c, int d) {
        if (c == kFirst) {
            const int k = d > 0 ? first_out : first_out - 1;
            first_out += d;
            if (k < run_below) u += 2 * d;
            return k >= run_below && k < run_below + len ? 0 : kNone;
        }
        const int k = d > 0 ? last_out : last_out - 1;
        last_out += d;
        return k < len - run_last ? run_last : kNone;
    };
    auto enter = [&](int c, bool runs) {
        u += c >> kBits;
        c &= kNone;
        if (runs && (c == kFirst || c == kLast)) c = in_run(c, 1);
        Mask bit;
        one_bit(bit, static_cast<unsigned>(c));
        out |= out + bit;
    };
    auto leave = [&](int c, bool runs) {
        u -= c >> kBits;
        c &= kNone;
        if (runs && (c == kFirst || c == kLast)) c = in_run(c, -1);
        Mask bit;
        one_bit(bit, static_cast<unsigned>(c));
        const Mask up = out & (~bit + 1);
        out ^= up & (~up + 1);
    };
    for (int r = 0; r < e; ++r) enter(r < n ? code[r * T] : kNone, runs);
    auto finish = [&](auto kind) {  // plain: no runs beyond the middle, five values kept always
        constexpr bool kPlain = decltype(kind)::value;
        int m = m_all;
        if (!kPlain)
            for (int r = 0; r < min(e, n); ++r) m -= value(r) != CUDART_INF_F;
#pragma unroll 2
        for (int r = 0; r < n; ++r) {
            leave(code[(r - 1 - e) * T], !kPlain && runs);
            enter(code[(r + e) * T], !kPlain && runs);
            const float v = value(r);
            double st = global;
            if (!kPlain) m += (r - 1 - e >= 0 && value(r - 1 - e) != CUDART_INF_F) - (r + e < n && value(r + e) != CUDART_INF_F);
            if (kPlain || m >= 5) {
                const Mask kept = all & ~out;
                const int plo = nth_bit(kept, (u - 1) >> 1, rows <= 15);
                const Mask above = kept & ~((static_cast<Mask>(2) << plo) - 1);
                const int phi = u & 1 ? plo : low_bit(above);
                // double add of the two middle values (preprocess.cpp:198)
                st = 0.5 * (static_cast<double>(S[plo * T]) + static_cast<double>(S[phi * T]));
            }
            residual[at[r]] = v != CUDART_INF_F ? __double2float_rn(static_cast<double>(v) - st) : CUDART_NAN_F;
        }
    };
    // (the warp takes one of the two)
    if (cg::coalesced_threads().any(runs || a.need - X < 5))
        finish(std::false_type());
    else
        finish(std::true_type());
}

// ------------------------------------------------------------------ samples + exact medians

// The regular sample grid of sample_pixels (common.hpp:85-100): every step-th
// column and row from `border`, finite values only, optionally masked. Order is
// irrelevant (only order statistics are taken); the count is exact. The image may
// be a band of a larger one: it holds the rows from oy on (row y at img + (y - oy) *
// pitch), and the grid is the whole image's, its rows border + (j0 + j) step for j <
// gh.
//
// Bound by memory, once the frame's counter is taken once for a CTA's 2048 points
// (one atomic a warp before: sampling and selection together 4.8 ms for 120 frames of
// 1030 x 777, now 0.75 ms).
constexpr int kSamplePoints = 8;  // of a thread

__global__ void __launch_bounds__(256) sample_kernel(const float* img, size_t plane, int pitch, int border, int step, int gw,
                                                     int j0, int gh, int oy, const float* mask, float* out, int cap,
                                                     int* counts) {
    __shared__ int warp_first[8];
    __shared__ int first;
    const int f = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned points = static_cast<unsigned>(gw) * static_cast<unsigned>(gh);  // at most 4 x 200000 (grid_step)
    const unsigned g0 = blockIdx.x * (256u * kSamplePoints) + threadIdx.x;
    float v[kSamplePoints];
    unsigned ok = 0;
#pragma unroll
    for (int i = 0; i < kSamplePoints; ++i) {
        const unsigned g = g0 + 256u * i;
        v[i] = CUDART_NAN_F;
        if (g < points) {
            const unsigned row = g / static_cast<unsigned>(gw);
            const int x = border + static_cast<int>(g - row * gw) * step;
            const int y = border + (j0 + static_cast<int>(row)) * step - oy;
            const size_t pix = static_cast<size_t>(y) * pitch + x;
            if (!mask || mask[pix] != 0.0f) v[i] = img[f * plane + pix];
        }
    }
    int mine = 0, before = 0;  // of this warp: its samples, and this thread's first
#pragma unroll
    for (int i = 0; i < kSamplePoints; ++i) {
        const unsigned b = __ballot_sync(0xffffffffu, finitef(v[i]));
        if (b >> lane & 1u) ok |= 1u << i;
        mine += __popc(b);
    }
    if (lane == 0) warp_first[warp] = mine;
    __syncthreads();
    if (threadIdx.x == 0) {
        int sum = 0;
        for (int k = 0; k < 8; ++k) {
            const int c = warp_first[k];
            warp_first[k] = sum;
            sum += c;
        }
        first = sum ? atomicAdd(&counts[f], sum) : 0;
    }
    __syncthreads();
    before = first + warp_first[warp];
#pragma unroll
    for (int i = 0; i < kSamplePoints; ++i) {
        const unsigned b = __ballot_sync(0xffffffffu, ok >> i & 1u);
        const int k = before + __popc(b & ((1u << lane) - 1u));
        if ((ok >> i & 1u) && k < cap) out[static_cast<size_t>(f) * cap + k] = v[i];
        before += __popc(b);
    }
}

inline void launch_sample(const float* img, size_t plane, int pitch, int n, int border, int step, int gw, int j0, int gh,
                          int oy, const float* mask, float* out, int cap, int* counts, cudaStream_t s) {
    const long long g = static_cast<long long>(gw) * gh, each = 256 * kSamplePoints;
    sample_kernel<<<dim3(static_cast<unsigned>((g + each - 1) / each), n), 256, 0, s>>>(img, plane, pitch, border, step, gw,
                                                                                      j0, gh, oy, mask, out, cap, counts);
    FTB_CHECK(cudaGetLastError());
}

__device__ __forceinline__ uint32_t order_key(float v) {
    const uint32_t b = __float_as_uint(v);
    return b ^ (static_cast<uint32_t>(static_cast<int>(b) >> 31) | 0x80000000u);
}
__device__ __forceinline__ float key_value(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// ---- exact order statistics of a frame's samples by a cluster of CTAs.
//
// The samples near the wanted rank are copied into shared memory, and radix passes
// over them (11 bits each, of the range that is left) find the value. Which are near
// comes from 1024 samples at regular places: the values 64 ranks on either side of
// theirs (four standard deviations of a random subset's) hold it, and an eighth of
// all samples. One pass over the samples then counts those below and collects those
// between. Where that misses (few distinct values overfill the lists, or an unlucky
// subset), the radix passes read all samples. Up to kSelAll samples are all kept.
//
// Bound by reading the samples once a median (two a sigma): an 8-bit radix select
// over all of them for either middle rank, 16 passes a sigma and most of their
// shared atomics on one of a few exponents' counters, measured 2.9 ms for 120 frames
// of 790,000 samples; sampling and this 4.8 ms then, 0.75 ms now.

constexpr int kSelCluster = 8;
constexpr int kSelThreads = 512;
constexpr int kSelList = 16384;  // keys a CTA keeps
constexpr int kSelBits = 11;
constexpr int kSelSubset = 1024;
constexpr int kSelSlack = 64;  // subset ranks on either side
constexpr int kSelAll = kSelCluster * kSelList;

struct SelShared {
    uint32_t list[kSelList];
    uint32_t hist[2][1 << kSelBits];
    uint32_t subset[kSelSubset];
    uint32_t bracket[2];
    int count, below;  // of this CTA: keys inside the bracket, below it
    uint32_t low;      // largest key below the result
    uint32_t warp_sum[kSelThreads / 32];
    uint32_t digit, before;
    int total[3];      // of the cluster: inside, below; whether a list overflowed
};

// MODE 0: keys of x; MODE 1: keys of float(|x - med|) (the MAD deviations,
// common.hpp:80).
template <int MODE>
__device__ __forceinline__ uint32_t sample_key(float v, double med) {
    if (MODE == 1) v = __double2float_rn(fabs(static_cast<double>(v) - med));
    return order_key(v);
}

// The median of cnt > 0 values, in every thread of the cluster: the value of rank
// cnt / 2 or, for an even count, its mean with the one before (common.hpp:64-76).
template <int MODE>
__device__ double cluster_median(const float* __restrict__ x, int cnt, double med, SelShared& sh) {
    cg::cluster_group cl = cg::this_cluster();
    const int rank = static_cast<int>(cl.block_rank()), t = static_cast<int>(threadIdx.x), lane = t & 31, warp = t >> 5;
    const int mid = cnt / 2;
    const bool even = cnt % 2 == 0;
    uint32_t lo = 0u, hi = 0xffffffffu;
    if (t == 0) {
        sh.count = sh.below = 0;
        sh.low = 0u;
    }
    for (int b = t; b < 2 << kSelBits; b += kSelThreads) sh.hist[0][b] = 0u;  // both
    if (cnt > kSelAll) {
        for (int q = t; q < kSelSubset; q += kSelThreads)
            sh.subset[q] = sample_key<MODE>(x[static_cast<long long>(q) * cnt / kSelSubset], med);
        __syncthreads();
        // the ranks of an eighth of the subset, four threads a value
        const int q = rank * (kSelSubset / kSelCluster) + (t >> 2);
        const uint32_t own = sh.subset[q];
        int r = 0;
        for (int e = t & 3; e < kSelSubset; e += 4) r += sh.subset[e] < own || (sh.subset[e] == own && e < q);
        r += __shfl_xor_sync(0xffffffffu, r, 1);
        r += __shfl_xor_sync(0xffffffffu, r, 2);
        const int mine = r == kSelSubset / 2 - kSelSlack ? 0 : r == kSelSubset / 2 + kSelSlack ? 1 : -1;
        if (mine >= 0 && (t & 3) == 0)
            for (int c = 0; c < kSelCluster; ++c) *cl.map_shared_rank(&sh.bracket[mine], c) = own;
        cl.sync();
        lo = sh.bracket[0];
        hi = sh.bracket[1];
    } else {
        __syncthreads();
    }
    // the keys between go to the list, those below are counted: eight a thread and
    // round, their places by one prefix sum and one atomic a warp (a ballot and an
    // atomic for each of them: 57 instructions a value, 0.70 ms for 120 frames of
    // 790,000, now 0.53)
    constexpr int kUnroll = 8, kChunk = kSelThreads * kUnroll;
    int below = 0;
    const uint32_t width = hi - lo;
    auto take = [&](const float* p, int left, auto whole) {
        constexpr bool kWhole = decltype(whole)::value;  // else only the values before `left`
        uint32_t key[kUnroll];
        unsigned in = 0;
#pragma unroll
        for (int i = 0; i < kUnroll; ++i) key[i] = __float_as_uint(kWhole || i * kSelThreads < left ? p[i * kSelThreads] : 0.0f);
#pragma unroll
        for (int i = 0; i < kUnroll; ++i) {
            const bool valid = kWhole || i * kSelThreads < left;
            key[i] = sample_key<MODE>(__uint_as_float(key[i]), med);
            if (valid && key[i] < lo) ++below;
            if (valid && key[i] - lo <= width) in |= 1u << i;
        }
        const int mine = __popc(in);
        int to = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, to, o);
            if (lane >= o) to += up;
        }
        int first = 0;
        if (lane == 31 && to) first = atomicAdd(&sh.count, to);
        to += __shfl_sync(0xffffffffu, first, 31) - mine;
#pragma unroll
        for (int i = 0; i < kUnroll; ++i)
            if (in >> i & 1u) {
                if (to < kSelList) sh.list[to] = key[i];
                ++to;
            }
    };
    for (int e0 = rank * kChunk; e0 < cnt; e0 += kChunk * kSelCluster) {
        if (e0 + kChunk <= cnt)
            take(x + e0 + t, 0, std::true_type());
        else
            take(x + e0 + t, cnt - e0 - t, std::false_type());
    }
    below = __reduce_add_sync(0xffffffffu, below);
    if (lane == 0 && below) atomicAdd(&sh.below, below);
    cl.sync();
    if (warp == 0) {
        int inside = 0, under = 0, over = 0;
        if (lane < kSelCluster) {
            inside = *cl.map_shared_rank(&sh.count, lane);
            under = *cl.map_shared_rank(&sh.below, lane);
            over = inside > kSelList;
        }
        inside = __reduce_add_sync(0xffffffffu, inside);
        under = __reduce_add_sync(0xffffffffu, under);
        over = __reduce_add_sync(0xffffffffu, over);
        if (lane == 0) {
            sh.total[0] = inside;
            sh.total[1] = under;
            sh.total[2] = over;
        }
    }
    __syncthreads();
    int k = mid - sh.total[1];  // rank among the keys that are looked at
    const bool listed = sh.total[2] == 0 && k - even >= 0 && k < sh.total[0];
    if (!listed) {
        lo = 0u;
        hi = 0xffffffffu;
        k = mid;
    }
    const int own = listed ? sh.count : 0;
    auto each = [&](auto&& f) {
        if (listed) {
            for (int e = t; e < own; e += kSelThreads) f(sh.list[e]);
        } else {
            for (int e = rank * kSelThreads + t; e < cnt; e += kSelThreads * kSelCluster) f(sample_key<MODE>(x[e], med));
        }
    };
    // radix passes over the keys in [base, base + 2^bits). Each counts into one
    // histogram and clears the other: a pass's are read after its barrier, and all
    // CTAs have read them when the next one's barrier is passed.
    uint32_t base = lo;
    int bits = 32 - __clz(hi - lo), flip = 0;
    while (bits > 0) {
        const int shift = max(0, bits - kSelBits);
        const uint32_t span = bits < 32 ? (1u << bits) - 1u : 0xffffffffu;
        uint32_t* hist = sh.hist[flip];
        each([&](uint32_t key) {
            const uint32_t d = key - base;
            if (key >= base && d <= span) atomicAdd(&hist[d >> shift], 1u);
        });
        cl.sync();
        // four digits a thread, summed over the cluster, and the one that holds rank k
        uint32_t sum[4] = {};
#pragma unroll
        for (int c = 0; c < kSelCluster; ++c) {
            const uint4 h = reinterpret_cast<const uint4*>(cl.map_shared_rank(hist, c))[t];
            sum[0] += h.x;
            sum[1] += h.y;
            sum[2] += h.z;
            sum[3] += h.w;
        }
        const uint32_t all = sum[0] + sum[1] + sum[2] + sum[3];
        uint32_t acc = all;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t up = __shfl_up_sync(0xffffffffu, acc, o);
            if (lane >= o) acc += up;
        }
        if (lane == 31) sh.warp_sum[warp] = acc;
        __syncthreads();
        for (int q = 0; q < warp; ++q) acc += sh.warp_sum[q];
        acc -= all;
        const uint32_t want = static_cast<uint32_t>(k);
        if (want >= acc && want < acc + all) {
            int d = 0;
            while (d < 3 && want >= acc + sum[d]) acc += sum[d++];
            sh.digit = static_cast<uint32_t>(4 * t + d);
            sh.before = acc;
        }
        flip ^= 1;
        for (int b = t; b < 1 << kSelBits; b += kSelThreads) sh.hist[flip][b] = 0u;
        __syncthreads();
        base += sh.digit << shift;
        k -= static_cast<int>(sh.before);
        bits = shift;
    }
    double m = key_value(base);
    if (even) {
        float lower = key_value(base);
        if (k == 0) {  // no equal one before: the largest key below
            uint32_t top = 0u;
            each([&](uint32_t key) {
                if (key < base) top = max(top, key);
            });
            top = __reduce_max_sync(0xffffffffu, top);
            if (lane == 0) atomicMax(&sh.low, top);
            cl.sync();
            for (int c = 0; c < kSelCluster; ++c) top = max(top, *cl.map_shared_rank(&sh.low, c));
            lower = key_value(top);
        }
        m = 0.5 * (m + lower);
    }
    cl.sync();  // all is read before the next median, or the end, takes the memory
    return m;
}

// sigma, or the median itself (MEDIAN), of a frame's samples: a cluster a frame
template <bool MEDIAN>
__global__ void __cluster_dims__(kSelCluster, 1, 1) __launch_bounds__(kSelThreads)
    select_kernel(const float* samples, int cap, const int* counts, double* out, int unit_if_zero) {
    extern __shared__ __align__(16) unsigned char sel[];
    SelShared& sh = *reinterpret_cast<SelShared*>(sel);
    const int f = blockIdx.x / kSelCluster;
    const int cnt = min(counts[f], cap);
    const float* x = samples + static_cast<size_t>(f) * cap;
    double r = 0.0;
    // every CTA of the cluster has started before any writes to another's shared memory
    cg::this_cluster().sync();
    if (MEDIAN) {
        if (cnt > 0) r = cluster_median<0>(x, cnt, 0.0, sh);
    } else {
        if (cnt >= 3) {
            const double med = cluster_median<0>(x, cnt, 0.0, sh);
            r = 1.4826 * cluster_median<1>(x, cnt, med, sh);
        }
        if (unit_if_zero && !(r > 0.0)) r = 1.0;
    }
    if (cg::this_cluster().block_rank() == 0 && threadIdx.x == 0) out[f] = r;
}

template <bool MEDIAN>
inline void launch_select(const float* samples, int cap, const int* counts, int n, double* out, int unit_if_zero,
                          cudaStream_t s) {
    allow_dynamic_smem(reinterpret_cast<const void*>(select_kernel<MEDIAN>), sizeof(SelShared));
    select_kernel<MEDIAN><<<n * kSelCluster, kSelThreads, sizeof(SelShared), s>>>(samples, cap, counts, out, unit_if_zero);
    FTB_CHECK(cudaGetLastError());
}

// ------------------------------------------------------------------ scatter + mask

struct ScatterArgs {
    const float* residual;
    const double* sigma;
    float* scatter;
    int w, h, pitch, n;
};

// scatter = 1.4826 * median_i float(|r_i| / sigma_i) over finite residuals, or
// 1e9 with fewer than n/2 of them (preprocess.cpp:380-389). The median's order
// statistics are found by counting (the values are >= 0, so their bit patterns
// order like the values).
__global__ void __launch_bounds__(128) scatter_kernel(const ScatterArgs a) {
    extern __shared__ unsigned char sm[];
    const int T = blockDim.x, t = threadIdx.x;
    uint32_t* C = reinterpret_cast<uint32_t*>(sm);
    const long long q = static_cast<long long>(blockIdx.x) * T + t;
    const int x = static_cast<int>(q % a.w), y = static_cast<int>(q / a.w);
    if (y >= a.h) return;
    const size_t plane = static_cast<size_t>(a.pitch) * a.h;
    const size_t pix = static_cast<size_t>(y) * a.pitch + x;
    int c = 0;
    for (int i = 0; i < a.n; ++i) {
        const float v = a.residual[i * plane + pix];
        if (!finitef(v)) continue;
        const float d = __double2float_rn(__ddiv_rn(static_cast<double>(fabsf(v)), a.sigma[i]));
        C[c * T + t] = __float_as_uint(d);
        ++c;
    }
    if (c < a.n / 2) {
        a.scatter[pix] = 1e9f;
        return;
    }
    const int mid = c / 2;
    uint32_t vmid = 0, vlow = 0;
    for (int e = 0; e < c; ++e) {
        const uint32_t ve = C[e * T + t];
        int less = 0, leq = 0;
        for (int f = 0; f < c; ++f) {
            const uint32_t vf = C[f * T + t];
            less += vf < ve;
            leq += vf <= ve;
        }
        if (less <= mid && mid < leq) vmid = ve;
        if (less <= mid - 1 && mid - 1 < leq) vlow = ve;
    }
    double m = __uint_as_float(vmid);
    if (c % 2 == 0) m = 0.5 * (m + __uint_as_float(vlow));
    a.scatter[pix] = __double2float_rn(1.4826 * m);
}

// a / b to nearest from r = 1 / b to nearest, for finite a >= 0 and b > 0 of a size
// that keeps quotient and remainders normal (a: a float, b: 1.4826 times one, or 1; the
// middle one of the deviations from a median does not exceed the largest float):
// the quotient by r is corrected once to within a unit in the last place, and by
// Markstein's theorem a second correction by its exact remainder rounds it correctly
// (P. W. Markstein, IBM J. Res. Develop. 34, 1990). Five operations for the general
// division's dozens.
__device__ __forceinline__ double quotient(double a, double b, double r) {
    double q = __dmul_rn(a, r);
    q = __fma_rn(__fma_rn(-b, q, a), r, q);
    return __fma_rn(__fma_rn(-b, q, a), r, q);
}

// The same for n <= N <= 128 by a sorting network in registers (Batcher's merge
// exchange) over the values' bit patterns (the values are >= +0.0 or +inf, so their
// patterns order like the values). The absent ones are zeros below and all-ones above
// such that the middle pair lies at N / 2 - 1 and N / 2: the exchanges that only
// order the rest are then not compiled.
//
// Bound by issue and the FP64 and conversion pipes; with the general division, a
// bitonic network of a power of two and the middle picked from all registers 40 frames
// of 2048^2 took 1.34 ms, now 0.36 (33 of 1501 x 1117: 0.48 -> 0.13).
template <int N>
__global__ void __launch_bounds__(N <= 64 ? 128 : 64) scatter_net_kernel(const ScatterArgs a) {
    __shared__ double2 sr[N];  // a frame's sigma and its reciprocal
    if (threadIdx.x < a.n) {
        const double sg = a.sigma[threadIdx.x];
        sr[threadIdx.x] = make_double2(sg, __drcp_rn(sg));
    }
    if (N > 64 && threadIdx.x + 64 < a.n) {
        const double sg = a.sigma[threadIdx.x + 64];
        sr[threadIdx.x + 64] = make_double2(sg, __drcp_rn(sg));
    }
    __syncthreads();
    constexpr int kSure = N <= 64 ? N - 8 : N - 16;  // launch_scatter takes the smallest network
    const unsigned q = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = static_cast<int>(q / static_cast<unsigned>(a.w)), x = static_cast<int>(q - y * static_cast<unsigned>(a.w));
    if (y >= a.h) return;
    const size_t plane = static_cast<size_t>(a.pitch) * a.h;
    const size_t pix = static_cast<size_t>(y) * a.pitch + x;
    const float* res = a.residual + pix;
    float v[N];
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = i < kSure || i < a.n ? __ldg(res + i * plane) : CUDART_NAN_F;
    int c = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) c += finitef(v[i]);
    if (c < a.n / 2 || c == 0) {  // (the median of no values is 0, with one frame)
        a.scatter[pix] = c < a.n / 2 ? 1e9f : 0.0f;
        return;
    }
    uint32_t sv[N];
    int low = N / 2 - c / 2;  // zeros still to come
#pragma unroll
    for (int i = 0; i < N; ++i) {
        if (finitef(v[i])) {
            sv[i] = __float_as_uint(__double2float_rn(quotient(static_cast<double>(fabsf(v[i])), sr[i].x, sr[i].y)));
        } else {
            sv[i] = low > 0 ? 0u : 0xffffffffu;
            --low;
        }
    }
#pragma unroll
    for (int p = 1; p < N; p <<= 1)
#pragma unroll
        for (int k = p; k > 0; k >>= 1)
#pragma unroll
            for (int i = 0; i < N; ++i)
                if (i >= k % p && i + k < N && ((i - k % p) / k) % 2 == 0 && i / (2 * p) == (i + k) / (2 * p)) {
                    const uint32_t lo = min(sv[i], sv[i + k]), hi = max(sv[i], sv[i + k]);
                    sv[i] = lo;
                    sv[i + k] = hi;
                }
    double m = __uint_as_float(sv[N / 2]);
    if (c % 2 == 0) m = 0.5 * (m + __uint_as_float(sv[N / 2 - 1]));
    a.scatter[pix] = __double2float_rn(1.4826 * m);
}

__global__ void mask_kernel(const float* scatter, float* mask, int w, int h, int pitch, int dil, double limit) {
    const long long q = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    const int x = static_cast<int>(q % w), y = static_cast<int>(q / w);
    if (y >= h) return;
    float out = 1.0f;
    for (int yy = max(0, y - dil); yy <= min(h - 1, y + dil) && out != 0.0f; ++yy)
        for (int xx = max(0, x - dil); xx <= min(w - 1, x + dil); ++xx)
            if (static_cast<double>(scatter[static_cast<size_t>(yy) * pitch + xx]) > limit) {
                out = 0.0f;
                break;
            }
    mask[static_cast<size_t>(y) * pitch + x] = out;
}

// ------------------------------------------------------------------ matched filter


struct FilterArgs {
    const float* residual;
    const float* mask;
    const float* scatter;
    const double* sigma;   // per-frame residual noise
    float* out;            // unnormalised filter output
    int* cr;               // cosmic-ray hits per frame
    const float* k;        // 2R+1 taps, float(exp(-i^2 / 2 s^2))
    float norm;            // float(1 / sum k^2)
    float wscat, hit, ratio, clip;
    int w, h, pitch, R;
};

// One CTA per (frame, 32 x 16 tile). z (normalised, weighted) over the tile plus
// a halo of R + 2; cosmic-ray centres over the tile plus R + 1; cleaned and
// clipped z over the tile plus R; then the horizontal pass over the tile's
// columns and the vertical pass. Pixels outside the image hold 0: a product with
// 0 adds +0.0f to a sum that starts at +0.0f, which equals the reference's
// truncated sums at the borders (preprocess.cpp:133-135, 140-145).
// Any radius: the filter of wide PSFs (filter_frames_kernel has the others).
__global__ void __launch_bounds__(256) filter_kernel(const FilterArgs a) {
    extern __shared__ float fs[];
    constexpr int TWc = 32, THc = 16;
    const int R = a.R, H = R + 2;
    const int ZW = TWc + 2 * H, ZH = THc + 2 * H;
    float* Z = fs;                                    // ZH x ZW  z, then cleaned z
    unsigned char* F = reinterpret_cast<unsigned char*>(Z + ZW * ZH);  // ZH x ZW cosmic-ray centre flags
    float* Tt = reinterpret_cast<float*>(F + ((ZW * ZH + 15) / 16) * 16);  // (THc + 2R) x TWc horizontal pass
    __shared__ int cr_tile;
    const int f = blockIdx.z;
    const int x0 = blockIdx.x * TWc, y0 = blockIdx.y * THc;
    const size_t plane = static_cast<size_t>(a.pitch) * a.h;
    const float inv = __double2float_rn(__ddiv_rn(1.0, a.sigma[f]));
    if (threadIdx.x == 0) cr_tile = 0;
    for (int e = threadIdx.x; e < ZW * ZH; e += blockDim.x) {
        const int gx = x0 - H + e % ZW, gy = y0 - H + e / ZW;
        float z = 0.0f;
        if (gx >= 0 && gy >= 0 && gx < a.w && gy < a.h) {
            // the three loads are independent, so they are in flight together
            const size_t pix = static_cast<size_t>(gy) * a.pitch + gx;
            const float v = __ldg(a.residual + f * plane + pix);
            const float mk = __ldg(a.mask + pix);
            const float s = __ldg(a.scatter + pix);
            if (mk != 0.0f && finitef(v)) {
                const float vm = __fmul_rn(v, inv);
                // (v / sigma) / e with e = scatter above weight_scatter, else 1 (an exact division)
                z = s > a.wscat ? __fdiv_rn(vm, s) : vm;
            }
        }
        Z[e] = z;
    }
    __syncthreads();
    // cosmic-ray centres (preprocess.cpp:433-447): inside [1, w-2] x [1, h-2]
    for (int e = threadIdx.x; e < ZW * ZH; e += blockDim.x) {
        const int lx = e % ZW, ly = e / ZW;
        const int gx = x0 - H + lx, gy = y0 - H + ly;
        unsigned char flag = 0;
        if (lx >= 1 && ly >= 1 && lx < ZW - 1 && ly < ZH - 1 && gx >= 1 && gy >= 1 && gx < a.w - 1 && gy < a.h - 1) {
            const float v = Z[e];
            if (v >= a.hit) {
                const float s4 = __fadd_rn(__fadd_rn(__fadd_rn(Z[e - 1], Z[e + 1]), Z[e - ZW]), Z[e + ZW]);
                const float n4 = __fmul_rn(0.25f, s4);
                if (!(n4 >= __fmul_rn(a.ratio, v))) {
                    flag = 1;
                    if (gx >= x0 && gx < x0 + TWc && gy >= y0 && gy < y0 + THc) atomicAdd(&cr_tile, 1);
                }
            }
        }
        F[e] = flag;
    }
    __syncthreads();
    // cleaned, clipped z over the tile plus R (kills applied after the scan)
    float* Zc = Z;  // in place: the kill test reads the original z of the same pixel only
    for (int e = threadIdx.x; e < ZW * ZH; e += blockDim.x) {
        const int lx = e % ZW, ly = e / ZW;
        if (lx < 2 || ly < 2 || lx >= ZW - 2 || ly >= ZH - 2) continue;
        const float v = Z[e];
        bool kill = F[e] != 0;
        if (!kill && v > 2.5f)
            for (int dy = -1; dy <= 1 && !kill; ++dy)
                for (int dx = -1; dx <= 1; ++dx)
                    if (F[e + dy * ZW + dx]) {
                        kill = true;
                        break;
                    }
        const float zc = kill ? 0.0f : v;
        const int gx = x0 - H + lx, gy = y0 - H + ly;
        // (outside the image 0 also where a negative clip would move it)
        Zc[e] = gx < 0 || gy < 0 || gx >= a.w || gy >= a.h ? 0.0f : zc < -a.clip ? -a.clip : (a.clip < zc ? a.clip : zc);
    }
    __syncthreads();
    // horizontal pass over rows y0-R .. y0+THc+R-1, the tile's columns
    const int TR = THc + 2 * R;
    for (int e = threadIdx.x; e < TR * TWc; e += blockDim.x) {
        const int c = e % TWc, r = e / TWc;
        const float* row = Zc + (r + 2) * ZW + (c + 2);  // centre column at H + c, row at 2 + r (= H - R + r)
        float acc = 0.0f;
        for (int j = 0; j <= 2 * R; ++j) acc = __fadd_rn(acc, __fmul_rn(row[j], a.k[j]));
        const int gy = y0 - R + r;
        Tt[e] = (gy >= 0 && gy < a.h) ? acc : 0.0f;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < TWc * THc; e += blockDim.x) {
        const int c = e % TWc, r = e / TWc;
        const int gx = x0 + c, gy = y0 + r;
        if (gx >= a.w || gy >= a.h) continue;
        float acc = 0.0f;
        // (the taps times the norm: the reference's float product)
        for (int j = 0; j <= 2 * R; ++j)
            acc = __fadd_rn(acc, __fmul_rn(__fmul_rn(a.k[j], a.norm), Tt[(r + j) * TWc + c]));
        a.out[f * plane + static_cast<size_t>(gy) * a.pitch + gx] = acc;
    }
    __syncthreads();
    if (threadIdx.x == 0 && cr_tile) atomicAdd(&a.cr[f], cr_tile);
}

template <int N, class Mask>
void launch_sky_middle(const SkyArgs& a, long long npix, cudaStream_t s) {
    constexpr int T = sky_threads(N);
    const size_t smem = 2 * sizeof(size_t) * a.n + static_cast<size_t>(T) *
        (4 * sky_rows(sky_middle(a.n, a.exclude)) + ((N <= 64 ? 4 : 0) + sizeof(typename SkyCode<Mask>::type)) * a.n +
         sizeof(typename SkyCode<Mask>::type) * (2 * std::min(a.exclude, a.n) + 1));
    auto kern = sky_middle_kernel<N, Mask>;
    allow_dynamic_smem(reinterpret_cast<const void*>(kern), smem);
    kern<<<static_cast<unsigned>((npix + T - 1) / T), T, smem, s>>>(a);
    FTB_CHECK(cudaGetLastError());
}

// Up to 128 frames the sort is a network of the next multiple of 8 or 16 values and the
// middle's mask the smallest that holds it (a longer window than the default one may
// need 64 or 128 bits, which only the 64- and 128-value networks are compiled for);
// more frames: rank counting.
void launch_sky(const SkyArgs& a, int n, long long npix, cudaStream_t s) {
    const int middle = sky_middle(n, a.exclude);
    if (n > 128 || npix > 0x7fffffffLL) {
        const int T = 64;
        const size_t smem = static_cast<size_t>(T) * n * 9;
        allow_dynamic_smem(reinterpret_cast<const void*>(sky_kernel), smem);
        sky_kernel<<<static_cast<unsigned>((npix + T - 1) / T), T, smem, s>>>(a);
        FTB_CHECK(cudaGetLastError());
    } else if (middle > 64) {
        launch_sky_middle<128, unsigned __int128>(a, npix, s);
    } else if (middle > 32) {
        n <= 64 ? launch_sky_middle<64, uint64_t>(a, npix, s) : launch_sky_middle<128, uint64_t>(a, npix, s);
    } else {
        switch (n <= 64 ? (n + 7) / 8 : 8 + (n - 64 + 15) / 16) {
            case 1: launch_sky_middle<8, uint32_t>(a, npix, s); break;
            case 2: launch_sky_middle<16, uint32_t>(a, npix, s); break;
            case 3: launch_sky_middle<24, uint32_t>(a, npix, s); break;
            case 4: launch_sky_middle<32, uint32_t>(a, npix, s); break;
            case 5: launch_sky_middle<40, uint32_t>(a, npix, s); break;
            case 6: launch_sky_middle<48, uint32_t>(a, npix, s); break;
            case 7: launch_sky_middle<56, uint32_t>(a, npix, s); break;
            case 8: launch_sky_middle<64, uint32_t>(a, npix, s); break;
            case 9: launch_sky_middle<80, uint32_t>(a, npix, s); break;
            case 10: launch_sky_middle<96, uint32_t>(a, npix, s); break;
            case 11: launch_sky_middle<112, uint32_t>(a, npix, s); break;
            default: launch_sky_middle<128, uint32_t>(a, npix, s); break;
        }
    }
}

template <int N>
void launch_scatter_net(const ScatterArgs& a, long long npix, cudaStream_t s) {
    constexpr int T = N <= 64 ? 128 : 64;
    scatter_net_kernel<N><<<static_cast<unsigned>((npix + T - 1) / T), T, 0, s>>>(a);
}

// the temporal scatter: the sorting network of the next multiple of 8 or 16 up to 128
// frames, counting beyond
void launch_scatter(const ScatterArgs& a, int n, long long npix, cudaStream_t s) {
    if (n <= 128 && npix <= 0x7fffffffLL) {
        switch (n <= 64 ? (n + 7) / 8 : 8 + (n - 64 + 15) / 16) {
            case 1: launch_scatter_net<8>(a, npix, s); break;
            case 2: launch_scatter_net<16>(a, npix, s); break;
            case 3: launch_scatter_net<24>(a, npix, s); break;
            case 4: launch_scatter_net<32>(a, npix, s); break;
            case 5: launch_scatter_net<40>(a, npix, s); break;
            case 6: launch_scatter_net<48>(a, npix, s); break;
            case 7: launch_scatter_net<56>(a, npix, s); break;
            case 8: launch_scatter_net<64>(a, npix, s); break;
            case 9: launch_scatter_net<80>(a, npix, s); break;
            case 10: launch_scatter_net<96>(a, npix, s); break;
            case 11: launch_scatter_net<112>(a, npix, s); break;
            default: launch_scatter_net<128>(a, npix, s); break;
        }
    } else {
        const int T = 128;
        const size_t smem = static_cast<size_t>(T) * n * 4;
        allow_dynamic_smem(reinterpret_cast<const void*>(scatter_kernel), smem);
        scatter_kernel<<<static_cast<unsigned>((npix + T - 1) / T), T, smem, s>>>(a);
    }
    FTB_CHECK(cudaGetLastError());
}

// 16-byte asynchronous copy global -> shared; a source outside the image copies
// nothing and fills zero (src-size 0).
__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool valid) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// The geometry of filter_frames_kernel for radius R: a 64 x TH tile whose horizontal
// pass has 62 or 64 rows, one item a thread; the residual tile with a halo of R + 2
// rows and of HA >= R + 2 columns, a multiple of four, so that its rows start at
// 16-byte boundaries.
template <int R>
struct FilterTile {
    static constexpr int TW = 64, TH = (64 - 2 * R) / 4 * 4, H = R + 2, HA = (R + 5) / 4 * 4;
    static constexpr int ZW = TW + 2 * HA, ZH = TH + 2 * H, ZN = ZW * ZH, TR = TH + 2 * R, FW = (ZW + 31) / 32;
    static constexpr int threads = 512;
    static constexpr size_t smem = sizeof(float) * (4 * ZN + TR * TW);
    static_assert(ZN % 4 == 0 && (TR / 2) * (TW / 4) <= threads && (TH / 4) * (TW / 2) <= threads && TR % 2 == 0, "one item a thread");
};

// The filter of filter_kernel for a run of frames per CTA (fixed radius R): the
// tile's mask and scatter weight are read once for all its frames (one float per pixel:
// NaN where masked, -1 outside the image, else the divisor, 1 for none), and the next
// frame's residual tile plus halo is copied asynchronously into a second buffer while
// the current one is filtered, so the loads of frame f + 1 overlap the arithmetic of
// frame f. Per frame the steps, their arithmetic and their order are filter_kernel's.
//
// Bound by issue: 40 of the slots of a pixel at R = 4 are the two passes' products and
// sums. The rest is kept short: four columns an item with 16-byte copies and shared
// loads, clipping in the pass that normalises, cosmic-ray centres as bits of which the
// neighbours are cleared only where a tile has one, and one double division a frame.
// One column an item, a flag byte a pixel and a cleaning pass over the tile took 286
// instructions a pixel, 1.89 ms for 40 frames of 2048^2 (R = 4) and 2.00 for 120 of 1030
// x 777 (R = 8); now 132, 0.81 and 0.67 ms.
template <int R>
__global__ void __launch_bounds__(FilterTile<R>::threads, 2) filter_frames_kernel(const FilterArgs a, int n, int fpc) {
    using G = FilterTile<R>;
    constexpr int TW = G::TW, TH = G::TH, H = G::H, HA = G::HA, ZW = G::ZW, ZH = G::ZH, ZN = G::ZN, TR = G::TR, FW = G::FW;
    constexpr int KN = 2 * R + 1;
    extern __shared__ __align__(16) float fs[];
    float* const Rb0 = fs;  // residual tile + halo, double-buffered
    float* const Rb1 = fs + ZN;
    float* E = fs + 2 * ZN;   // weight divisor, NaN: masked, -1: outside
    float* Z = fs + 3 * ZN;   // cleaned and clipped z
    float* Tt = fs + 4 * ZN;  // TR x TW horizontal pass
    __shared__ uint32_t centre[ZH * FW];  // cosmic-ray centres
    __shared__ float inverse[256];        // float(1 / sigma) of the run's frames
    float kk[KN], kp[KN];  // the taps, and the taps times the norm (the reference's float product)
#pragma unroll
    for (int j = 0; j < KN; ++j) {
        kk[j] = a.k[j];
        kp[j] = __fmul_rn(kk[j], a.norm);
    }
    const int x0 = blockIdx.x * TW, y0 = blockIdx.y * TH;
    const int fa = blockIdx.z * fpc, fb = min(n, fa + fpc);
    const size_t plane = static_cast<size_t>(a.pitch) * a.h;
    const int tid = threadIdx.x;
    auto issue = [&](float* dst, int f) {
        const float* base = a.residual + f * plane;
        for (int e = tid; e < ZN / 4; e += G::threads) {
            const int gx = x0 - HA + 4 * (e % (ZW / 4)), gy = y0 - H + e / (ZW / 4);
            const bool in = gx >= 0 && gy >= 0 && gx < a.w && gy < a.h;  // (columns beyond w: the row's padding)
            cp_async16(dst + 4 * e, in ? base + static_cast<size_t>(gy) * a.pitch + gx : base, in);
        }
        cp_async_commit();
    };
    if (fa < fb) issue(Rb0, fa);
    for (int e = tid; e < ZN; e += G::threads) {
        const int gx = x0 - HA + e % ZW, gy = y0 - H + e / ZW;
        float ev = -1.0f;
        if (gx >= 0 && gy >= 0 && gx < a.w && gy < a.h) {
            const size_t pix = static_cast<size_t>(gy) * a.pitch + gx;
            const float mk = __ldg(a.mask + pix), sc = __ldg(a.scatter + pix);
            ev = mk != 0.0f ? (sc > a.wscat ? sc : 1.0f) : CUDART_NAN_F;  // (a scatter is not negative)
        }
        E[e] = ev;
    }
    for (int e = tid; e < ZH * FW; e += G::threads) centre[e] = 0u;
    if (tid < fb - fa) inverse[tid] = __double2float_rn(__ddiv_rn(1.0, a.sigma[fa + tid]));
    auto clipped = [&](float z) { return z < -a.clip ? -a.clip : (a.clip < z ? a.clip : z); };
    for (int f = fa; f < fb; ++f) {
        const float* cur = ((f - fa) & 1) ? Rb1 : Rb0;
        cp_async_wait_all();
        __syncthreads();  // cur is complete; every thread is past its last read of the other buffer
        if (f + 1 < fb) issue(((f - fa) & 1) ? Rb0 : Rb1, f + 1);
        const float inv = inverse[f - fa];
        // z: (v / sigma) / weight, 0 where masked, outside or not finite
        auto zval = [&](float v, float ev) {
            float z = 0.0f;
            if (ev >= 0.0f && finitef(v)) {
                const float vm = __fmul_rn(v, inv);
                // (v / sigma) / e, e = scatter above weight_scatter, else 1 (an exact division)
                z = ev != 1.0f ? __fdiv_rn(vm, ev) : vm;
            }
            return z;
        };
        auto zat = [&](int e) { return zval(cur[e], E[e]); };
        // z over the tile + R + 2, clipped, and in the same pass the cosmic-ray centres
        // (preprocess.cpp:433-447, inside [1, w-2] x [1, h-2]): a z at or above
        // the hit level takes its four neighbours' z from the residual tile
        // (the same arithmetic as their own entries)
        bool any = false;
        for (int e4 = tid; e4 < ZN / 4; e4 += G::threads) {
            const float4 v = reinterpret_cast<const float4*>(cur)[e4], ev = reinterpret_cast<const float4*>(E)[e4];
            float4 z, cz;
            if (ev.x == 1.0f && ev.y == 1.0f && ev.z == 1.0f && ev.w == 1.0f) {
                z.x = finitef(v.x) ? __fmul_rn(v.x, inv) : 0.0f;
                z.y = finitef(v.y) ? __fmul_rn(v.y, inv) : 0.0f;
                z.z = finitef(v.z) ? __fmul_rn(v.z, inv) : 0.0f;
                z.w = finitef(v.w) ? __fmul_rn(v.w, inv) : 0.0f;
                cz = make_float4(clipped(z.x), clipped(z.y), clipped(z.z), clipped(z.w));
            } else {
                z = make_float4(zval(v.x, ev.x), zval(v.y, ev.y), zval(v.z, ev.z), zval(v.w, ev.w));
                cz = make_float4(ev.x < 0.0f ? 0.0f : clipped(z.x), ev.y < 0.0f ? 0.0f : clipped(z.y),
                                 ev.z < 0.0f ? 0.0f : clipped(z.z), ev.w < 0.0f ? 0.0f : clipped(z.w));
            }
            if (z.x >= a.hit || z.y >= a.hit || z.z >= a.hit || z.w >= a.hit) {
                const int ly = e4 / (ZW / 4), lx0 = 4 * (e4 % (ZW / 4)), gy = y0 - H + ly;
                for (int c = 0; c < 4; ++c) {
                    const float zc = c == 0 ? z.x : c == 1 ? z.y : c == 2 ? z.z : z.w;
                    const int lx = lx0 + c, gx = x0 - HA + lx;
                    if (!(zc >= a.hit) || lx < HA - R - 1 || lx >= HA + TW + R + 1 || ly < 1 || ly >= ZH - 1 || gx < 1 ||
                        gy < 1 || gx >= a.w - 1 || gy >= a.h - 1)
                        continue;
                    const int e = 4 * e4 + c;
                    const float s4 = __fadd_rn(__fadd_rn(__fadd_rn(zat(e - 1), zat(e + 1)), zat(e - ZW)), zat(e + ZW));
                    const float n4 = __fmul_rn(0.25f, s4);
                    if (!(n4 >= __fmul_rn(a.ratio, zc))) {
                        atomicOr(&centre[ly * FW + (lx >> 5)], 1u << (lx & 31));
                        any = true;
                    }
                }
            }
            reinterpret_cast<float4*>(Z)[e4] = cz;
        }
        if (__syncthreads_or(any)) {
            // the centres, and their neighbours above 2.5, are cleared (after the scan)
            int inside = 0;
            for (int q = tid; q < ZH * FW; q += G::threads) {
                uint32_t bits = centre[q];
                centre[q] = 0u;
                const int ly = q / FW;
                while (bits) {
                    const int lx = 32 * (q % FW) + __ffs(static_cast<int>(bits)) - 1;
                    bits &= bits - 1u;
                    const int gx = x0 - HA + lx, gy = y0 - H + ly;
                    inside += gx >= x0 && gx < x0 + TW && gy >= y0 && gy < y0 + TH;
                    for (int dy = -1; dy <= 1; ++dy)
                        for (int dx = -1; dx <= 1; ++dx) {
                            const int e = (ly + dy) * ZW + lx + dx;
                            if ((dx == 0 && dy == 0) || zat(e) > 2.5f) Z[e] = clipped(0.0f);
                        }
                }
            }
            if (inside) atomicAdd(&a.cr[f], inside);
            __syncthreads();
        }
        // horizontal pass over rows y0-R .. y0+TH+R-1, the tile's columns: rows
        // in pairs (r, r + 1) and CQ adjacent columns per item; the pair's two
        // products of a tap are scalar round-to-nearest multiplies and their adds
        // into the pair's sums one __fadd2_rn (each output the reference's row[j]
        // * k[j] added in tap order), and the CQ columns share the loaded row
        // segments. The products stay scalar: a paired multiply followed by a
        // paired add was contracted into a fused multiply-add by the compiler
        // (even from inline PTX mul.rn.f32x2, and with --fmad=false), which rounds
        // once and differs from the reference in the last bits.
        if (tid < (TR / 2) * (TW / 4)) {
            constexpr int CQ = 4, OFF = HA - R, SKIP = OFF % 4, NQ = (SKIP + CQ + KN - 1 + 3) / 4;
            const int c = (tid % (TW / CQ)) * CQ, r = 2 * (tid / (TW / CQ));
            const float4* r0 = reinterpret_cast<const float4*>(Z + (r + 2) * ZW + c + OFF - SKIP);
            float2 v[4 * NQ];
#pragma unroll
            for (int x = 0; x < NQ; ++x) {
                const float4 p = r0[x], q = r0[x + ZW / 4];
                v[4 * x] = make_float2(p.x, q.x);
                v[4 * x + 1] = make_float2(p.y, q.y);
                v[4 * x + 2] = make_float2(p.z, q.z);
                v[4 * x + 3] = make_float2(p.w, q.w);
            }
            float2 acc[CQ];
#pragma unroll
            for (int q = 0; q < CQ; ++q) {
                acc[q] = make_float2(0.0f, 0.0f);
#pragma unroll
                for (int j = 0; j < KN; ++j)
                    acc[q] = __fadd2_rn(acc[q], make_float2(__fmul_rn(v[SKIP + q + j].x, kk[j]), __fmul_rn(v[SKIP + q + j].y, kk[j])));
            }
            float4* to = reinterpret_cast<float4*>(Tt + r * TW + c);
            to[0] = make_float4(acc[0].x, acc[1].x, acc[2].x, acc[3].x);  // (rows outside the image: sums of zeros)
            to[TW / 4] = make_float4(acc[0].y, acc[1].y, acc[2].y, acc[3].y);
        }
        __syncthreads();
        // vertical pass: two adjacent columns (one 8-byte load of the horizontal
        // pass) and RQ rows per item, the loaded column pairs shared by the rows
        if (tid < (TH / 4) * (TW / 2)) {
            constexpr int RQ = 4, NV = RQ + KN - 1;
            const int c = 2 * (tid % (TW / 2)), r = (tid / (TW / 2)) * RQ;
            const int gx = x0 + c;
            if (gx < a.w) {
                float* out = a.out + f * plane + static_cast<size_t>(y0 + r) * a.pitch + gx;
                float2 tv[NV];
#pragma unroll
                for (int x = 0; x < NV; ++x) tv[x] = *reinterpret_cast<const float2*>(Tt + (r + x) * TW + c);
#pragma unroll
                for (int q = 0; q < RQ; ++q) {
                    if (y0 + r + q >= a.h) break;
                    float2 acc = make_float2(0.0f, 0.0f);
#pragma unroll
                    for (int j = 0; j < KN; ++j)
                        acc = __fadd2_rn(acc, make_float2(__fmul_rn(kp[j], tv[q + j].x), __fmul_rn(kp[j], tv[q + j].y)));
                    float* o = out + static_cast<size_t>(q) * a.pitch;
                    if (gx + 1 < a.w) {
                        *reinterpret_cast<float2*>(o) = acc;
                    } else {
                        o[0] = acc.x;
                    }
                }
            }
        }
    }
}

template <int R>
void launch_filter_frames(const FilterArgs& a, int n, int sms, cudaStream_t s) {
    using G = FilterTile<R>;
    const int tx = (a.w + G::TW - 1) / G::TW, ty = (a.h + G::TH - 1) / G::TH;
    // frames split over CTAs until there are four waves of two CTAs an SM (at fewer the
    // last one's idle SMs cost more than reading mask and scatter again)
    const long long tiles = static_cast<long long>(tx) * ty;
    const int groups = static_cast<int>(std::min<long long>(n, std::max<long long>(1, (8LL * sms + tiles - 1) / tiles)));
    const int fpc = (n + groups - 1) / groups;
    auto kern = filter_frames_kernel<R>;
    allow_dynamic_smem(reinterpret_cast<const void*>(kern), G::smem);
    kern<<<dim3(tx, ty, (n + fpc - 1) / fpc), G::threads, G::smem, s>>>(a, n, fpc);
    FTB_CHECK(cudaGetLastError());
}

void launch_filter(const FilterArgs& a, int n, cudaStream_t s) {
    constexpr int TWc = 32, THc = 16;
    const int R = a.R, H = R + 2, ZW = TWc + 2 * H, ZH = THc + 2 * H;
    const size_t smem = sizeof(float) * ZW * ZH + ((ZW * ZH + 15) / 16) * 16 + sizeof(float) * (THc + 2 * R) * TWc;
    allow_dynamic_smem(reinterpret_cast<const void*>(filter_kernel), smem);
    filter_kernel<<<dim3((a.w + TWc - 1) / TWc, (a.h + THc - 1) / THc, n), 256, smem, s>>>(a);
    FTB_CHECK(cudaGetLastError());
}

void launch_filter_any(const FilterArgs& a, int n, int sms, cudaStream_t s) {
    switch (a.R) {
        case 1: launch_filter_frames<1>(a, n, sms, s); break;
        case 2: launch_filter_frames<2>(a, n, sms, s); break;
        case 3: launch_filter_frames<3>(a, n, sms, s); break;
        case 4: launch_filter_frames<4>(a, n, sms, s); break;
        case 5: launch_filter_frames<5>(a, n, sms, s); break;
        case 6: launch_filter_frames<6>(a, n, sms, s); break;
        case 7: launch_filter_frames<7>(a, n, sms, s); break;
        case 8: launch_filter_frames<8>(a, n, sms, s); break;
        default: launch_filter(a, n, s); break;
    }
}

// Bound by memory: each thread scales four columns of four rows (one pixel a thread
// with a 64-bit division for its row: 595 us for 40 frames of 2048^2, 2.3 TB/s; now
// 193 us).
//
// to: where the scaled frames go, rows to_pitch floats apart (g itself, or a caller's
// buffer of any alignment: the copy out of the stage's own layout, 0.42 ms for those
// frames, is this pass's stores).
__global__ void __launch_bounds__(256) rescale_kernel(const float* g, size_t plane, int w, int h, int pitch, const double* sg,
                                                      float* to, int to_pitch) {
    const int f = blockIdx.z;
    const double s = sg[f];
    const bool scale = s > 0.0;
    if (!scale && to == g) return;
    const float ig = scale ? __double2float_rn(__ddiv_rn(1.0, s)) : 0.0f;
    auto times = [&](float v) { return scale ? __fmul_rn(v, ig) : v; };
    const bool quads = to_pitch % 4 == 0 && reinterpret_cast<uintptr_t>(to) % 16 == 0;
    const int x = 4 * static_cast<int>(blockIdx.y * 64 + (threadIdx.x & 63)), y0 = static_cast<int>(blockIdx.x * 16 + (threadIdx.x >> 6));
    if (x >= w) return;
    const float* p = g + f * plane + static_cast<size_t>(y0) * pitch + x;
    float* o = to + f * (static_cast<size_t>(to_pitch) * h) + static_cast<size_t>(y0) * to_pitch + x;
    const size_t down = 4 * static_cast<size_t>(pitch), to_down = 4 * static_cast<size_t>(to_pitch);
    float4 v[4];  // (columns beyond w: the row's padding, not stored)
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (y0 + 4 * k < h) v[k] = *reinterpret_cast<const float4*>(p + k * down);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (y0 + 4 * k >= h) break;
        const float4 r = make_float4(times(v[k].x), times(v[k].y), times(v[k].z), times(v[k].w));
        float* q = o + k * to_down;
        if (quads && x + 3 < w) {
            *reinterpret_cast<float4*>(q) = r;
        } else {
            q[0] = r.x;
            if (x + 1 < w) q[1] = r.y;
            if (x + 2 < w) q[2] = r.z;
            if (x + 3 < w) q[3] = r.w;
        }
    }
}

// (rows along the grid's x, which has no limit of 65,535)
inline void launch_rescale(const float* g, size_t plane, int w, int h, int pitch, int n, const double* sg, float* to,
                           int to_pitch, cudaStream_t s) {
    rescale_kernel<<<dim3((h + 15) / 16, (w + 255) / 256, n), 256, 0, s>>>(g, plane, w, h, pitch, sg, to, to_pitch);
    FTB_CHECK(cudaGetLastError());
}

// v -> float(v - bg), NaN stays NaN (preprocess.cpp:235), then the blank areas grown
// by kGrow pixels: NaN wherever a non-finite value lies within +-kGrow in x and y
// (preprocess.cpp:240-253). in and out: bases and rows at 16-byte boundaries.
//
// A CTA takes 128 x 32 pixels and the kGrow rows above and below; a lane holds four
// columns, its non-finite ones as four bits that spread over the neighbours' by
// shuffles, and down the columns through a byte a lane and row in shared memory. Bound
// by memory (subtraction in place and 49 loads a pixel in a second kernel: 1.43 ms for
// 33 frames of 1501 x 1117, 0.44 GB; now 156 us).
constexpr int kGrow = 3;
constexpr int kPrepRows = 32;

__global__ void __launch_bounds__(256) subtract_grow_kernel(const float* __restrict__ in, float* __restrict__ out, size_t plane,
                                                            int w, int h, int pitch, const double* bg) {
    static_assert(kGrow <= 4, "a lane's neighbours reach four columns");
    constexpr int R = kPrepRows + 2 * kGrow, K = (R + 7) / 8;
    __shared__ unsigned char bad[R][32];
    const int f = blockIdx.z, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int x = static_cast<int>(blockIdx.y) * 128 + 4 * lane, y0 = static_cast<int>(blockIdx.x) * kPrepRows;
    const double b = bg[f];
    const float* src = in + f * plane;
    // four columns of a row and the bits of the non-finite ones; columns outside the image are not
    auto load = [&](int xx, int yy, float4& v) {
        const float4 r = *reinterpret_cast<const float4*>(src + static_cast<size_t>(yy) * pitch + xx);
        auto sub = [&](float q) { return finitef(q) ? __double2float_rn(static_cast<double>(q) - b) : CUDART_NAN_F; };
        v = make_float4(sub(r.x), sub(r.y), sub(r.z), sub(r.w));
        const unsigned m = (finitef(v.x) ? 0u : 1u) | (finitef(v.y) ? 0u : 2u) | (finitef(v.z) ? 0u : 4u) | (finitef(v.w) ? 0u : 8u);
        return xx + 3 < w ? m : m & ((1u << (w - xx)) - 1u);
    };
    float4 v[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int row = warp + 8 * k, y = y0 - kGrow + row;
        if (row >= R) break;
        unsigned m = 0, edge = 0;
        if (y >= 0 && y < h) {
            float4 beside;
            if (x < w) m = load(x, y, v[k]);
            if (lane == 0 && x > 0) edge = load(x - 4, y, beside);
            if (lane == 31 && x + 4 < w) edge = load(x + 4, y, beside);
        }
        unsigned left = __shfl_up_sync(0xffffffffu, m, 1), right = __shfl_down_sync(0xffffffffu, m, 1);
        if (lane == 0) left = edge;
        if (lane == 31) right = edge;
        unsigned d = left | m << 4 | right << 8;
        unsigned wide = d;
#pragma unroll
        for (int c = 1; c <= kGrow; ++c) wide |= d << c | d >> c;
        bad[row][lane] = static_cast<unsigned char>(wide >> 4 & 15u);
    }
    __syncthreads();
    if (x >= w) return;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int row = warp + 8 * k, y = y0 - kGrow + row;
        if (row < kGrow || row >= kPrepRows + kGrow || y >= h) continue;
        unsigned m = 0;
#pragma unroll
        for (int c = -kGrow; c <= kGrow; ++c) m |= bad[row + c][lane];
        const float4 r = make_float4(m & 1u ? CUDART_NAN_F : v[k].x, m & 2u ? CUDART_NAN_F : v[k].y,
                                     m & 4u ? CUDART_NAN_F : v[k].z, m & 8u ? CUDART_NAN_F : v[k].w);
        float* p = out + f * plane + static_cast<size_t>(y) * pitch + x;
        if (x + 3 < w) {
            *reinterpret_cast<float4*>(p) = r;
        } else {
            p[0] = r.x;
            if (x + 1 < w) p[1] = r.y;
            if (x + 2 < w) p[2] = r.z;
        }
    }
}

inline void launch_subtract_grow(const float* in, float* out, size_t plane, int w, int h, int pitch, int n, const double* bg,
                                 cudaStream_t s) {
    subtract_grow_kernel<<<dim3((h + kPrepRows - 1) / kPrepRows, (w + 127) / 128, n), 256, 0, s>>>(in, out, plane, w, h,
                                                                                                    pitch, bg);
    FTB_CHECK(cudaGetLastError());
}

inline int grid_step(int w, int h, int border, size_t max_samples) {
    const size_t usable = static_cast<size_t>(std::max(0, w - 2 * border)) * static_cast<size_t>(std::max(0, h - 2 * border));
    if (usable == 0) return 0;
    return std::max(1, static_cast<int>(std::sqrt(static_cast<double>(usable) / static_cast<double>(max_samples))));
}

inline int grid_count(int lo, int hi, int step) { return hi <= lo ? 0 : (hi - lo + step - 1) / step; }

}  // namespace

// ------------------------------------------------------------------ host driver

void stage_time_ranks(const double* t_h, int n, std::vector<int>& rank) {
    // stable sort of the frame indices by time (preprocess.cpp:323-331)
    std::vector<int> order(static_cast<size_t>(n));
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return t_h[a] < t_h[b]; });
    rank.assign(static_cast<size_t>(n), 0);
    for (int r = 0; r < n; ++r) rank[static_cast<size_t>(order[static_cast<size_t>(r)])] = r;
}

int sample_grid_points(int w, int h, int border) {
    const int st = grid_step(w, h, border, 200000);
    return st > 0 ? grid_count(border, w - border, st) * grid_count(border, h - border, st) : 0;
}

int filter_border(double fwhm_px) { return static_cast<int>(std::ceil(3 * fwhm_px * kFwhmToSigma)) + 1; }

StageScratch::StageScratch(Context& c, int w, int h, int n, double fwhm_px) : w_(w), h_(h), n_(n) {
    const int pitch = frame_pitch(w);
    const size_t plane = static_cast<size_t>(pitch) * h;
    residual = DevBuf(&c, sizeof(float) * plane * n, "residuals");
    scatter = DevBuf(&c, sizeof(float) * plane, "scatter map");
    // room for any sample grid this stage can use (borders 0 .. 64, and the PSF's)
    cap = std::max(1, sample_grid_points(w, h, filter_border(fwhm_px)));
    for (int b = 0; b <= 64; ++b) cap = std::max(cap, sample_grid_points(w, h, b));
    samples = DevBuf(&c, sizeof(float) * static_cast<size_t>(cap) * n, "noise samples");
    small = DevBuf(&c, 4096 + sizeof(double) * 2 * n + sizeof(int) * 2 * n + static_cast<size_t>(n), "stage tables");
}

bool StageScratch::fits(int w, int h, int n, double fwhm_px) const {
    return w == w_ && h == h_ && n == n_ && sample_grid_points(w, h, filter_border(fwhm_px)) <= cap;
}

bool StageScratch::holds(int w, int h, int n) const { return w == w_ && h <= h_ && n == n_; }

// The device tables of a stage in StageScratch::small: filter taps, per-frame
// sigma, filter sigma, sample counts, cosmic-ray tallies, the frame of each time rank.
struct StageTables {
    float* taps;
    double* sigma;
    double* sg;
    int* counts;
    int* cr;
    unsigned char* frame_of;
};

static StageTables stage_tables(StageScratch& sc, int n) {
    unsigned char* base = sc.small.as<unsigned char>();
    StageTables t;
    t.taps = reinterpret_cast<float*>(base);  // up to 512 floats
    t.sigma = reinterpret_cast<double*>(base + 2048);
    t.sg = t.sigma + n;
    t.counts = reinterpret_cast<int*>(t.sg + n);
    t.cr = t.counts + n;
    t.frame_of = reinterpret_cast<unsigned char*>(t.cr + n);
    return t;
}

void stage_noise(Context& c, StageScratch& sc, const float* d_sub, int w, int h, int n, const double* t_h,
                 int static_exclude, float* d_sky, int sub_pitch) {
    if (n < 1 || n > 255) throw std::runtime_error("stage: between 1 and 255 frames are supported");
    if (w != sc.w_ || h != sc.h_ || n != sc.n_) throw std::runtime_error("stage: scratch sized for another shape");
    const int pitch = frame_pitch(w);
    const size_t plane = static_cast<size_t>(pitch) * h;
    const long long npix = static_cast<long long>(w) * h;
    cudaStream_t s = c.stream();
    const StageTables tb = stage_tables(sc, n);

    // the frame of each time rank
    std::vector<int> rank;
    stage_time_ranks(t_h, n, rank);
    const int exclude = static_exclude >= 0 ? static_exclude : std::max(1, static_cast<int>(std::lround(n / 8.0)));
    std::vector<unsigned char> frame_of(static_cast<size_t>(n));
    for (int i = 0; i < n; ++i) frame_of[static_cast<size_t>(rank[static_cast<size_t>(i)])] = static_cast<unsigned char>(i);
    FTB_CHECK(cudaMemcpyAsync(tb.frame_of, frame_of.data(), frame_of.size(), cudaMemcpyHostToDevice, s));
    FTB_CHECK(cudaMemsetAsync(tb.counts, 0, sizeof(int) * 2 * n, s));  // counts and cosmic-ray tallies
    // 1. static sky + residuals
    {
        const int span = c.span_begin("static sky + residuals");
        SkyArgs a{d_sub, sc.residual.as<float>(), d_sky, tb.frame_of, w, h, pitch, n, exclude,
                  std::max(5, static_cast<int>(0.6 * n)), sub_pitch > 0 ? sub_pitch : pitch};
        launch_sky(a, n, npix, s);
        ++c.launches;
        c.span_end(span);
    }
    // 2. per-frame noise from the residual samples (border 2)
    {
        const int span = c.span_begin("noise");
        const int st = grid_step(w, h, 2, 200000);
        if (st > 0) {
            const int gw = grid_count(2, w - 2, st), gh = grid_count(2, h - 2, st);
            launch_sample(sc.residual.as<float>(), plane, pitch, n, 2, st, gw, 0, gh, 0, nullptr, sc.samples.as<float>(),
                          sc.cap, tb.counts, s);
            ++c.launches;
        }
        launch_select<false>(sc.samples.as<float>(), sc.cap, tb.counts, n, tb.sigma, 1, s);
        ++c.launches;
        c.span_end(span);
    }
}

void stage_filter(Context& c, StageScratch& sc, int w, int h, int n, const StageParams& sp, float* d_filtered,
                  float* d_mask, double* h_sigma, int* h_cr, float* d_out, int out_pitch) {
    if (!sc.fits(w, h, n, sp.fwhm_px)) throw std::runtime_error("stage: scratch sized for another shape");
    const int pitch = frame_pitch(w);
    const size_t plane = static_cast<size_t>(pitch) * h;
    const long long npix = static_cast<long long>(w) * h;
    cudaStream_t s = c.stream();
    const StageTables tb = stage_tables(sc, n);
    // the separable filter taps (preprocess.cpp:118-126)
    const double psf_sigma = sp.fwhm_px * kFwhmToSigma;
    const int R = std::max(1, static_cast<int>(std::ceil(3.0 * psf_sigma)));
    std::vector<float> taps(static_cast<size_t>(2 * R + 1));
    double k2 = 0.0;
    for (int i = -R; i <= R; ++i) {
        const double v = std::exp(-0.5 * i * i / (psf_sigma * psf_sigma));
        taps[static_cast<size_t>(i + R)] = static_cast<float>(v);
        k2 += v * v;
    }
    if (taps.size() > 512) throw std::runtime_error("stage: PSF too wide");
    FTB_CHECK(cudaMemcpyAsync(tb.taps, taps.data(), sizeof(float) * taps.size(), cudaMemcpyHostToDevice, s));
    float* d_taps = tb.taps;
    double* d_sigma = tb.sigma;
    double* d_sg = tb.sg;
    int* d_counts = tb.counts;
    int* d_cr = tb.cr;
    // 3. scatter map and mask
    {
        const int span = c.span_begin("scatter mask");
        ScatterArgs a{sc.residual.as<float>(), d_sigma, sc.scatter.as<float>(), w, h, pitch, n};
        launch_scatter(a, n, npix, s);
        ++c.launches;
        const int dil = std::max(1, static_cast<int>(std::lround(0.5 * sp.fwhm_px)));
        mask_kernel<<<static_cast<unsigned>((npix + 255) / 256), 256, 0, s>>>(sc.scatter.as<float>(), d_mask, w, h,
                                                                              pitch, dil, sp.mask_scatter);
        FTB_CHECK(cudaGetLastError());
        ++c.launches;
        c.span_end(span);
    }
    // 4. normalise, cosmic rays, clip, matched filter
    {
        const int span = c.span_begin("matched filter");
        FilterArgs a;
        a.residual = sc.residual.as<float>();
        a.mask = d_mask;
        a.scatter = sc.scatter.as<float>();
        a.sigma = d_sigma;
        a.out = d_filtered;
        a.cr = d_cr;
        a.k = d_taps;
        a.norm = static_cast<float>(1.0 / k2);
        a.wscat = static_cast<float>(sp.weight_scatter);
        a.hit = static_cast<float>(sp.cr_sigma);
        a.ratio = static_cast<float>(0.5 * std::exp(-0.5 / (psf_sigma * psf_sigma)));
        a.clip = static_cast<float>(sp.clip_sigma);
        a.w = w;
        a.h = h;
        a.pitch = pitch;
        a.R = R;
        launch_filter_any(a, n, c.sms(), s);
        ++c.launches;
        c.span_end(span);
    }
    // 5. robust sigma of the masked filter output (border ceil(3 s) + 1), rescale
    {
        const int span = c.span_begin("filter normalisation");
        const int fb = static_cast<int>(std::ceil(3 * psf_sigma)) + 1;
        FTB_CHECK(cudaMemsetAsync(d_counts, 0, sizeof(int) * n, s));
        const int st = grid_step(w, h, fb, 200000);
        if (st > 0) {
            const int gw = grid_count(fb, w - fb, st), gh = grid_count(fb, h - fb, st);
            if (static_cast<long long>(gw) * gh > sc.cap) throw std::runtime_error("stage: sample buffer too small");
            launch_sample(d_filtered, plane, pitch, n, fb, st, gw, 0, gh, 0, d_mask, sc.samples.as<float>(), sc.cap,
                          d_counts, s);
            ++c.launches;
        }
        launch_select<false>(sc.samples.as<float>(), sc.cap, d_counts, n, d_sg, 0, s);
        ++c.launches;
        launch_rescale(d_filtered, plane, w, h, pitch, n, d_sg, d_out ? d_out : d_filtered, d_out ? out_pitch : pitch, s);
        ++c.launches;
        c.span_end(span);
    }
    if (h_sigma) FTB_CHECK(cudaMemcpyAsync(h_sigma, d_sigma, sizeof(double) * n, cudaMemcpyDeviceToHost, s));
    if (h_cr) FTB_CHECK(cudaMemcpyAsync(h_cr, d_cr, sizeof(int) * n, cudaMemcpyDeviceToHost, s));
}

void stage_run(Context& c, StageScratch& sc, const float* d_sub, int w, int h, int n, const double* t_h,
               const StageParams& sp, float* d_filtered, float* d_sky, float* d_mask, double* h_sigma, int* h_cr,
               int sub_pitch, float* d_out, int out_pitch) {
    stage_noise(c, sc, d_sub, w, h, n, t_h, sp.static_exclude, d_sky, sub_pitch);
    stage_filter(c, sc, w, h, n, sp, d_filtered, d_mask, h_sigma, h_cr, d_out, out_pitch);
}

void stage_sigma_to_host(Context& c, StageScratch& sc, int n, double* h_sigma) {
    FTB_CHECK(cudaMemcpyAsync(h_sigma, stage_tables(sc, n).sigma, sizeof(double) * n, cudaMemcpyDeviceToHost,
                              c.stream()));
}

void prepare_sub(Context& c, StageScratch& sc, const float* d_raw, float* d_sub, int w, int h, int n, double* h_bg) {
    const int pitch = frame_pitch(w);
    const size_t plane = static_cast<size_t>(pitch) * h;
    cudaStream_t s = c.stream();
    const StageTables tb = stage_tables(sc, n);
    const int span = c.span_begin("background + borders");
    FTB_CHECK(cudaMemsetAsync(tb.counts, 0, sizeof(int) * n, s));
    const int st = grid_step(w, h, 0, 200000);
    if (st > 0) {
        const int gw = grid_count(0, w, st), gh = grid_count(0, h, st);
        launch_sample(d_raw, plane, pitch, n, 0, st, gw, 0, gh, 0, nullptr, sc.samples.as<float>(), sc.cap, tb.counts, s);
        ++c.launches;
    }
    launch_select<true>(sc.samples.as<float>(), sc.cap, tb.counts, n, tb.sg, 0, s);
    ++c.launches;
    launch_subtract_grow(d_raw, d_sub, plane, w, h, pitch, n, tb.sg, s);
    ++c.launches;
    c.span_end(span);
    if (h_bg) FTB_CHECK(cudaMemcpyAsync(h_bg, tb.sg, sizeof(double) * n, cudaMemcpyDeviceToHost, s));
}

// ------------------------------------------------------------------ bands (the tiled search)

void stage_sky(Context& c, StageScratch& sc, const float* d_sub, int w, int rows, int n, const double* t_h,
               int static_exclude, float* d_sky) {
    if (!sc.holds(w, rows, n)) throw std::runtime_error("stage: scratch sized for another shape");
    const int pitch = frame_pitch(w);
    const long long npix = static_cast<long long>(w) * rows;
    cudaStream_t s = c.stream();
    const StageTables tb = stage_tables(sc, n);
    std::vector<int> rank;
    stage_time_ranks(t_h, n, rank);
    const int exclude = static_exclude >= 0 ? static_exclude : std::max(1, static_cast<int>(std::lround(n / 8.0)));
    std::vector<unsigned char> frame_of(static_cast<size_t>(n));
    for (int i = 0; i < n; ++i) frame_of[static_cast<size_t>(rank[static_cast<size_t>(i)])] = static_cast<unsigned char>(i);
    FTB_CHECK(cudaMemcpyAsync(tb.frame_of, frame_of.data(), frame_of.size(), cudaMemcpyHostToDevice, s));
    const int span = c.span_begin("static sky + residuals");
    SkyArgs a{d_sub, sc.residual.as<float>(), d_sky, tb.frame_of, w, rows, pitch, n, exclude,
              std::max(5, static_cast<int>(0.6 * n)), pitch};
    launch_sky(a, n, npix, s);
    ++c.launches;
    c.span_end(span);
}

void sample_band(Context& c, const float* d_img, size_t plane, int pitch, int n, int w, int h, int border, int oy,
                 int core_y0, int core_y1, const float* d_mask, float* d_samples, int cap, int* d_counts) {
    const int st = grid_step(w, h, border, 200000);
    if (st <= 0) return;
    const int gw = grid_count(border, w - border, st);
    // the whole image's grid rows border + j st (< h - border) inside the core
    const int lo = std::max(core_y0, border), hi = std::min(core_y1, h - border);
    if (hi <= lo) return;
    const int j0 = (lo - border + st - 1) / st;
    const int j1 = (hi - border + st - 1) / st;
    const int gh = j1 - j0;
    if (gh <= 0 || gw <= 0) return;
    launch_sample(d_img, plane, pitch, n, border, st, gw, j0, gh, oy, d_mask, d_samples, cap, d_counts, c.stream());
    ++c.launches;
}

void select_sigma(Context& c, const float* d_samples, int cap, const int* d_counts, int n, double* d_out,
                  int unit_if_zero) {
    launch_select<false>(d_samples, cap, d_counts, n, d_out, unit_if_zero, c.stream());
    ++c.launches;
}

void select_median(Context& c, const float* d_samples, int cap, const int* d_counts, int n, double* d_out) {
    launch_select<true>(d_samples, cap, d_counts, n, d_out, 0, c.stream());
    ++c.launches;
}

void sample_frames(Context& c, const float* d_frames, size_t plane, int pitch, int n, int w, int h, int border,
                   float* d_samples, int cap, int* d_counts) {
    const int st = grid_step(w, h, border, 200000);
    if (st <= 0) return;
    const int gw = grid_count(border, w - border, st), gh = grid_count(border, h - border, st);
    const long long g = static_cast<long long>(gw) * gh;
    if (g > cap) throw std::runtime_error("sample_frames: sample buffer too small");
    launch_sample(d_frames, plane, pitch, n, border, st, gw, 0, gh, 0, nullptr, d_samples, cap, d_counts, c.stream());
    ++c.launches;
}

void subtract_grow(Context& c, const float* d_raw, float* d_sub, int w, int rows, int n, const double* d_bg) {
    const int pitch = frame_pitch(w);
    const size_t plane = static_cast<size_t>(pitch) * rows;
    launch_subtract_grow(d_raw, d_sub, plane, w, rows, pitch, n, d_bg, c.stream());
    ++c.launches;
}

void stage_filter_given(Context& c, StageScratch& sc, int w, int rows, int n, const StageParams& sp,
                        const double* d_sigma, const double* d_sg, float* d_filtered, float* d_mask) {
    if (!sc.holds(w, rows, n)) throw std::runtime_error("stage: scratch sized for another shape");
    const int pitch = frame_pitch(w);
    const size_t plane = static_cast<size_t>(pitch) * rows;
    const long long npix = static_cast<long long>(w) * rows;
    cudaStream_t s = c.stream();
    const StageTables tb = stage_tables(sc, n);
    const double psf_sigma = sp.fwhm_px * kFwhmToSigma;
    const int R = std::max(1, static_cast<int>(std::ceil(3.0 * psf_sigma)));
    std::vector<float> taps(static_cast<size_t>(2 * R + 1));
    double k2 = 0.0;
    for (int i = -R; i <= R; ++i) {
        const double v = std::exp(-0.5 * i * i / (psf_sigma * psf_sigma));
        taps[static_cast<size_t>(i + R)] = static_cast<float>(v);
        k2 += v * v;
    }
    if (taps.size() > 512) throw std::runtime_error("stage: PSF too wide");
    FTB_CHECK(cudaMemcpyAsync(tb.taps, taps.data(), sizeof(float) * taps.size(), cudaMemcpyHostToDevice, s));
    {
        const int span = c.span_begin("scatter mask");
        ScatterArgs a{sc.residual.as<float>(), d_sigma, sc.scatter.as<float>(), w, rows, pitch, n};
        launch_scatter(a, n, npix, s);
        const int dil = std::max(1, static_cast<int>(std::lround(0.5 * sp.fwhm_px)));
        mask_kernel<<<static_cast<unsigned>((npix + 255) / 256), 256, 0, s>>>(sc.scatter.as<float>(), d_mask, w, rows,
                                                                              pitch, dil, sp.mask_scatter);
        FTB_CHECK(cudaGetLastError());
        c.launches += 2;
        c.span_end(span);
    }
    {
        const int span = c.span_begin("matched filter");
        FTB_CHECK(cudaMemsetAsync(tb.cr, 0, sizeof(int) * n, s));
        FilterArgs a;
        a.residual = sc.residual.as<float>();
        a.mask = d_mask;
        a.scatter = sc.scatter.as<float>();
        a.sigma = d_sigma;
        a.out = d_filtered;
        a.cr = tb.cr;
        a.k = tb.taps;
        a.norm = static_cast<float>(1.0 / k2);
        a.wscat = static_cast<float>(sp.weight_scatter);
        a.hit = static_cast<float>(sp.cr_sigma);
        a.ratio = static_cast<float>(0.5 * std::exp(-0.5 / (psf_sigma * psf_sigma)));
        a.clip = static_cast<float>(sp.clip_sigma);
        a.w = w;
        a.h = rows;
        a.pitch = pitch;
        a.R = R;
        launch_filter_any(a, n, c.sms(), s);
        ++c.launches;
        c.span_end(span);
    }
    if (d_sg) {
        launch_rescale(d_filtered, plane, w, rows, pitch, n, d_sg, d_filtered, pitch, s);
        ++c.launches;
    }
}

void frame_sample_stats(Context& c, const float* const* d_frames, int k, int w, int h, int pitch, float* d_samples,
                        int cap, int* d_counts, double* d_stats) {
    cudaStream_t s = c.stream();
    FTB_CHECK(cudaMemsetAsync(d_counts, 0, sizeof(int) * k, s));
    const int st = grid_step(w, h, 0, 200000);
    if (st > 0) {
        const int gw = grid_count(0, w, st), gh = grid_count(0, h, st);
        const long long g = static_cast<long long>(gw) * gh;
        if (g > cap) throw std::runtime_error("frame_sample_stats: sample buffer too small");
        for (int i = 0; i < k; ++i) {
            launch_sample(d_frames[i], 0, pitch, 1, 0, st, gw, 0, gh, 0, nullptr, d_samples + static_cast<size_t>(i) * cap,
                          cap, d_counts + i, s);
            ++c.launches;
        }
    }
    launch_select<true>(d_samples, cap, d_counts, k, d_stats, 0, s);
    launch_select<false>(d_samples, cap, d_counts, k, d_stats + k, 0, s);
    c.launches += 2;
}

}  // namespace ftb
