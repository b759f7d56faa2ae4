// Legacy-ASCII VTK output formatted on the GPU.
//
// The reference writes every field value with `ofstream << float`
// (src/moment_vtk_writer.cu:8-48): the float, widened to double, printed as
// printf "%g" with precision 6 (six significant digits, round-half-even on the
// exact binary value, trailing zeros removed, exponent form below 1e-4 and from
// 1e6 up).  fmt_g6 produces those bytes with integer arithmetic only, so the
// host and the device builds give the same text; a CPU test checks it against
// the C library's printf.
//
// A field of N cells becomes N lines ("v\n", "|u|\n" or "u v w\n").  One kernel,
// vtk_emit: a block takes 256 lines, finds each value's six digits and exponent
// once (g6_parse), which give the line lengths, gets its place in the text from
// the blocks before it by looking back over their published lengths, writes the
// characters (g6_put) to shared memory where they belong, and stores the block's
// text with 4-byte words.  Blocks number themselves in the order they start, so a
// block only ever waits for blocks that are already running.
//
// lbm_vtk_writer runs the whole snapshot asynchronously: the kernels are
// queued on the caller's stream (ordered after the step that produced the
// fields), and a writer thread copies the text to pinned host memory in chunks
// on its own stream and writes the file while the solver keeps stepping.
#include <cuda_runtime.h>

#include <condition_variable>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <deque>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "lbm_capi.h"
#include "lbm_internal.h"

#define HD __host__ __device__ __forceinline__

namespace lbm {
void set_error(const std::string& msg);
namespace vtk {

// ---- exact "%g" (precision 6) of a float --------------------------------

// unsigned integer of 6 little-endian 32-bit limbs (192 bits: the largest
// product formed below, n * 2^149 with n < 2^21, needs 170)
struct Big {
    uint32_t w[6];
};

HD void big_set(Big& a, uint64_t v) {
    a.w[0] = (uint32_t)v;
    a.w[1] = (uint32_t)(v >> 32);
    a.w[2] = a.w[3] = a.w[4] = a.w[5] = 0;
}

HD void big_mul(Big& a, uint32_t k) {
    uint64_t c = 0;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        const uint64_t t = (uint64_t)a.w[i] * k + c;
        a.w[i] = (uint32_t)t;
        c = t >> 32;
    }
}

HD void big_mul_pow5(Big& a, int k) {
    while (k >= 13) {
        big_mul(a, 1220703125u);   // 5^13
        k -= 13;
    }
    uint32_t p = 1;
    for (int i = 0; i < k; ++i) p *= 5u;
    big_mul(a, p);
}

HD void big_shl(Big& a, int s) {
    const int l = s >> 5, b = s & 31;
    for (int i = 5; i >= 0; --i) {
        const int j = i - l;
        uint32_t hi = j >= 0 ? a.w[j] : 0u;
        uint32_t lo = j - 1 >= 0 ? a.w[j - 1] : 0u;
        a.w[i] = b ? (hi << b) | (lo >> (32 - b)) : hi;
    }
}

HD int big_cmp(const Big& a, const Big& b) {
    for (int i = 5; i >= 0; --i)
        if (a.w[i] != b.w[i]) return a.w[i] < b.w[i] ? -1 : 1;
    return 0;
}

HD void big_sub(Big& a, const Big& b) {
    uint64_t borrow = 0;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        const uint64_t t = (uint64_t)a.w[i] - b.w[i] - borrow;
        a.w[i] = (uint32_t)t;
        borrow = (t >> 63) & 1u;
    }
}

// floor(v * 10^s) for v = m * 2^e as n, with the rest compared to one half:
// half = -1 below, 0 exactly, +1 above.  The value is A / D with
// s >= 0: A = m 5^s 2^max(t,0), D = 2^max(-t,0); s < 0: A = m 2^max(t,0),
// D = 5^-s 2^max(-t,0); t = e + s.  n starts from a double estimate and is
// corrected by exact comparisons.
HD uint32_t scaled_floor(uint32_t m, int e, int s, int& half) {
    const int t = e + s;
    Big A, D;
    big_set(A, m);
    big_set(D, 1);
    if (s >= 0) big_mul_pow5(A, s);
    else big_mul_pow5(D, -s);
    if (t >= 0) big_shl(A, t);
    else big_shl(D, -t);
    // estimate: v * 10^s in double (only a starting point)
    double est = ldexp((double)m, e);
    for (int k = s; k > 0; --k) est *= 10.0;
    for (int k = s; k < 0; ++k) est /= 10.0;
    uint32_t n = est < 1.0 ? 0u : (est > 4.0e9 ? 4000000000u : (uint32_t)est);
    Big nD;
    for (;;) {   // the largest n with n D <= A
        nD = D;
        big_mul(nD, n);
        if (big_cmp(nD, A) > 0) { --n; continue; }
        Big n1;  // (n + 1) D = n D + D
        uint64_t c = 0;
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            const uint64_t x = (uint64_t)nD.w[i] + D.w[i] + c;
            n1.w[i] = (uint32_t)x;
            c = x >> 32;
        }
        if (big_cmp(n1, A) <= 0) { ++n; continue; }
        break;
    }
    Big R = A;
    big_sub(R, nD);
    big_shl(R, 1);
    half = big_cmp(R, D);
    return n;
}

// 10^k for 0 <= k <= 22, all exact doubles
#define G6_POW10                                                                                                   \
    {1e0, 1e1, 1e2, 1e3, 1e4, 1e5, 1e6, 1e7, 1e8, 1e9, 1e10, 1e11, 1e12, 1e13, 1e14, 1e15, 1e16, 1e17, 1e18, 1e19, \
     1e20, 1e21, 1e22}

// A value as printf("%g") shows it: its six digits (a byte each, the first in the
// lowest byte), decimal exponent x, sign, and kind 0 (a number), 1 (zero), 2 (inf),
// 3 (nan); last: index of the last digit kept (trailing zeros are dropped).
struct G6 {
    uint64_t d;
    int8_t x;
    uint8_t neg, kind, last;
};

// six digits of n < 10^6, a byte each, the first in the lowest byte
HD uint64_t g6_digits(uint32_t n) {
    const uint32_t hi = n / 1000u, lo = n - hi * 1000u;
    auto three = [](uint32_t v) {      // v < 1000
        const uint32_t a = v / 100u, r = v - a * 100u, b = r / 10u;
        return a | (b << 8) | ((r - b * 10u) << 16);
    };
    return (uint64_t)three(hi) | ((uint64_t)three(lo) << 24);
}

// the digits by exact integer comparison: values next to a rounding or digit boundary
__host__ __device__ __noinline__ void g6_exact(uint32_t m, int e, int& X, uint32_t& n, int& half) {
    for (int it = 0; it < 4; ++it) {
        n = scaled_floor(m, e, 5 - X, half);
        if (n >= 1000000u) { ++X; continue; }
        if (n < 100000u) { --X; continue; }
        break;
    }
}

// p10: the powers of ten (shared memory on the device)
HD G6 g6_parse(float v, const double* p10) {
    G6 g{};
    uint32_t bits;
    memcpy(&bits, &v, 4);
    g.neg = (uint8_t)(bits >> 31);
    const uint32_t E = (bits >> 23) & 0xffu, F = bits & 0x7fffffu;
    if (E == 0xffu) { g.kind = F ? 3 : 2; return g; }
    if (E == 0 && F == 0) { g.kind = 1; return g; }
    const uint32_t m = E ? (F | 0x800000u) : F;
    const int e = (E ? (int)E : 1) - 150;
    // decimal exponent: floor(log10 v), from the bit length, then corrected
#ifdef __CUDA_ARCH__
    const int b = 32 - __clz((int)m);
#else
    const int b = 32 - __builtin_clz(m);
#endif
    const int l2 = b - 1 + e;                                  // floor(log2 v)
    int X = (l2 >= 0) ? (l2 * 78913) >> 18 : -((-l2 * 78913 + 262143) >> 18);   // ~ l2 * log10(2)
    uint32_t n = 0;
    int half = 0;
    // fast path: y = v 10^k in double with one correctly rounded operation
    // (10^|k| is exact for |k| <= 22), so |y - exact| <= 2^-33 for y < 2^20;
    // taken only when floor(y) and the side of one half are certain (y is exact,
    // or far enough from both), else the exact path below decides
    const double x = (double)(bits >> 31 ? -v : v);
    bool done = false;
    // the estimate is X or X - 1: settle it by comparison where both powers are at hand
    if (X >= -16 && X <= 4 && x * p10[5 - X] >= 1000000.0) ++X;
    for (int it = 0; it < 3; ++it) {
        const int k = 5 - X;
        if (k < -22 || k > 22) break;
        const double p = p10[k < 0 ? -k : k];
        const double y = k >= 0 ? x * p : x / p;
        if (y >= 1000000.0) { ++X; continue; }
        if (y < 100000.0) { --X; continue; }
        const uint32_t fl = (uint32_t)y;
        const double fr = y - (double)fl, tol = 0x1p-30;
        const bool exact = k >= 0 && fma(x, p, -y) == 0.0;
        if (!exact && (fr < tol || fr > 1.0 - tol || fabs(fr - 0.5) < tol)) break;
        n = fl;
        half = fr > 0.5 ? 1 : (fr < 0.5 ? -1 : 0);
        done = true;
        break;
    }
    if (!done) {
        int xe = X, he = 0;
        uint32_t ne = 0;
        g6_exact(m, e, xe, ne, he);      // (its results by address: X, n and half stay in registers)
        X = xe; n = ne; half = he;
    }
    if (half > 0 || (half == 0 && (n & 1u))) {
        if (++n == 1000000u) { n = 100000u; ++X; }
    }
    g.d = g6_digits(n);
    g.x = (int8_t)X;
#ifdef __CUDA_ARCH__
    g.last = (uint8_t)((63 - __clzll((long long)g.d)) >> 3);
#else
    g.last = (uint8_t)((63 - __builtin_clzll(g.d)) >> 3);
#endif
    return g;
}

// number of characters of g
HD int g6_len(const G6& g) {
    const int neg = g.neg;
    if (g.kind) return neg + (g.kind == 1 ? 1 : 3);
    const int X = g.x, last = g.last;
    if (X < -4 || X >= 6) return neg + 1 + (last > 0 ? last + 1 : 0) + 4;
    if (X >= 0) return neg + X + 1 + (last > X ? 1 + last - X : 0);
    return neg + 2 + (-X - 1) + last + 1;
}

// up to 16 characters, the first in the lowest byte of lo
struct Text {
    uint64_t lo, hi;
    int len;
};
// the k characters of v behind those of t (k <= 8; v holds nothing above them)
HD void text_add(Text& t, uint64_t v, int k) {
    if (t.len < 8) {
        t.lo |= v << (8 * t.len);
        if (t.len > 0) t.hi |= v >> (64 - 8 * t.len);
    } else {
        t.hi |= v << (8 * (t.len - 8));
    }
    t.len += k;
}

// the characters of g, at most 12: [-] digits with a point behind digit x (0 in
// exponent form, or "0." and zeros in front of all), [e+dd]
HD Text g6_text(const G6& g) {
    Text t{0, 0, 0};
    if (g.neg) text_add(t, '-', 1);
    if (g.kind) {
        if (g.kind == 1) text_add(t, '0', 1);
        else text_add(t, g.kind == 3 ? 0x6e616eull : 0x666e69ull, 3);      // "nan", "inf"
        return t;
    }
    const int X = g.x, last = g.last;
    const uint64_t dg = g.d + 0x303030303030ull;
    const bool ex = X < -4 || X >= 6;
    const int point = ex ? 0 : X;
    if (point < 0) {
        text_add(t, 0x3030302e30ull & ((1ull << (8 * (1 - point))) - 1), 1 - point);      // "0." and -X-1 zeros
        text_add(t, dg & ((1ull << (8 * (last + 1))) - 1), last + 1);
    } else {
        const int in = point + 1;                                          // digits before the point
        const uint64_t low = dg & ((1ull << (8 * in)) - 1);
        if (last > point) {
            const uint64_t frac = (dg >> (8 * in)) & ((1ull << (8 * (last - point))) - 1);
            text_add(t, low | ((uint64_t)'.' << (8 * in)) | (frac << (8 * (in + 1))), last + 2);
        } else {
            text_add(t, low, in);
        }
        if (ex) {
            const int a = X < 0 ? -X : X, tens = a / 10;
            text_add(t, 'e' | ((X < 0 ? '-' : '+') << 8) | ((uint64_t)('0' + tens) << 16) |
                            ((uint64_t)('0' + a - 10 * tens) << 24), 4);
        }
    }
    return t;
}

// Bytes of printf("%g", (double)v) into out (at most 12); returns the length.
inline int fmt_g6(float v, char* out) {
    static const double p10[23] = G6_POW10;
    const Text t = g6_text(g6_parse(v, p10));
    for (int i = 0; i < t.len; ++i) out[i] = (char)((i < 8 ? t.lo >> (8 * i) : t.hi >> (8 * (i - 8))) & 0xff);
    return t.len;
}

// |u| exactly as speed_kernel computes it (the same expression)
__device__ __forceinline__ float speed3(float u, float v, float w) {
    const float uu = u * u + v * v + w * w;
    return sqrtf(uu);
}

constexpr int LINES = 256;           // lines per block
constexpr int MAXLINE = 39;          // "u v w\n" at 12 bytes per value

__device__ const double kPow10[23] = G6_POW10;

// Place of a block in the text: state[k] of block k is LEN | its bytes once they
// are known, SUM | the bytes of blocks 0 .. k once those are.  One warp looks back,
// 32 blocks at a time, until it finds a SUM.  The wait is bounded: every block
// looked at has started, so a wait that runs out means that the launch is broken;
// the block then publishes BAD, as do all behind it, and writes nothing.
constexpr uint64_t LEN = 1ull << 62, SUM = 2ull << 62, BAD = 3ull << 62, VAL = LEN - 1;
constexpr int kPolls = 1 << 22;

__device__ __forceinline__ uint64_t state_ld(const uint64_t* p) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void state_st(uint64_t* p, uint64_t v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// called by one whole warp once the block has published its length (block 0: its sum); returns the bytes before block `me`, or BAD
__device__ uint64_t text_place(uint64_t* state, int64_t me, uint32_t total) {
    const int lane = threadIdx.x & 31;
    if (me == 0) return 0;
    uint64_t before = 0;
    for (int64_t end = me; end > 0;) {          // blocks end-32 .. end-1 are looked at, lane 0 the nearest
        const int64_t j = end - 1 - lane;
        uint64_t v = SUM;                        // (before the first block: a sum of nothing)
        int polls = 0;
        if (j >= 0)
            while ((v = state_ld(state + j)) < LEN && ++polls < kPolls) __nanosleep(20);
        const uint64_t kind = v & BAD;
        if (__any_sync(0xffffffffu, kind == 0 || kind == BAD)) {
            if (lane == 0) state_st(state + me, BAD);
            return BAD;
        }
        const uint32_t sums = __ballot_sync(0xffffffffu, kind == SUM);
        const int stop = sums ? __ffs((int)sums) - 1 : 32;      // the nearest sum ends the walk
        uint64_t add = lane <= stop ? (v & VAL) : 0;
        for (int o = 16; o; o >>= 1) add += __shfl_xor_sync(0xffffffffu, add, o);
        before += add;
        if (sums) break;
        end -= 32;
    }
    if (lane == 0) state_st(state + me, SUM | (before + total));
    return before;
}

// Bound by issue slots: about 440 instructions a value (a third of them integer
// multiplies, shifts and tests of the digits and the text), against 4-12 B read and
// 8-35 B written a line.  u v w of 256x128x128 cells (4.19 M lines): 242 us, from 452
// in the two-kernel form that formatted every value twice through arrays in local
// memory; looking back before the text is made, instead of behind it, 315 us.
template <int KIND>
__global__ void __launch_bounds__(LINES, 4) vtk_emit(const float* a, const float* b, const float* c, int64_t n,
                                                  uint32_t* ticket, uint64_t* state, int64_t nb, char* text) {
    constexpr int NV = KIND == LBM_VTK_VECTOR ? 3 : 1;
    __shared__ __align__(16) char stage[LINES * (KIND == LBM_VTK_VECTOR ? MAXLINE : 13) + 16];
    __shared__ uint32_t ws[LINES / 32];
    __shared__ uint32_t block;
    __shared__ uint64_t place;
    __shared__ double p10[23];
    if (threadIdx.x == 0) block = atomicAdd(ticket, 1u);
    if (threadIdx.x < 23) p10[threadIdx.x] = kPow10[threadIdx.x];
    __syncthreads();
    const int64_t me = block;
    const int64_t i = me * LINES + threadIdx.x;
    G6 g[NV];
    uint32_t len = 0;
    if (i < n) {
        if (KIND == LBM_VTK_SCALAR) {
            g[0] = g6_parse(a[i], p10);
        } else if (KIND == LBM_VTK_SPEED) {
            g[0] = g6_parse(speed3(a[i], b[i], c[i]), p10);
        } else {
            const float v[3] = {a[i], b[i], c[i]};
#pragma unroll
            for (int k = 0; k < NV; ++k) g[k] = g6_parse(v[k], p10);
        }
#pragma unroll
        for (int k = 0; k < NV; ++k) len += (uint32_t)g6_len(g[k]) + 1u;      // a blank or the line's end behind each
    }
    // exclusive scan of the line lengths inside the block
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t s = len;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += y;
    }
    if (lane == 31) ws[warp] = s;
    __syncthreads();
    uint32_t wbase = 0, total = 0;
    for (int k = 0; k < LINES / 32; ++k) {
        if (k < warp) wbase += ws[k];
        total += ws[k];
    }
    if (threadIdx.x == 0) state_st(state + me, (me == 0 ? SUM : LEN) | total);
    // the line's characters in words: whole words are stored as such, and a word that the
    // line shares with its neighbours byte by byte
    if (i < n) {
        uint32_t at = wbase + s - len;
        uint64_t acc = 0;
        uint32_t fill = at & 3u;              // bytes of the current word before and in acc
        uint32_t skip = fill;                 // of them, the neighbour's
        uint32_t* w = reinterpret_cast<uint32_t*>(stage) + (at >> 2);
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            Text t = g6_text(g[k]);
            text_add(t, k == NV - 1 ? '\n' : ' ', 1);
            const uint32_t part[4] = {(uint32_t)t.lo, (uint32_t)(t.lo >> 32), (uint32_t)t.hi, (uint32_t)(t.hi >> 32)};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int m = min(max(t.len - 4 * j, 0), 4);
                acc |= (uint64_t)part[j] << (8u * fill);
                fill += (uint32_t)m;
                if (fill >= 4u) {
                    if (skip) {
                        char* o = reinterpret_cast<char*>(w);
                        for (uint32_t q = skip; q < 4u; ++q) o[q] = (char)(acc >> (8u * q));
                        skip = 0;
                    } else {
                        *w = (uint32_t)acc;
                    }
                    ++w;
                    acc >>= 32;
                    fill -= 4u;
                }
            }
        }
        char* o = reinterpret_cast<char*>(w);
        for (uint32_t q = skip; q < fill; ++q) o[q] = (char)(acc >> (8u * q));
    }
    if (warp == 0) {
        const uint64_t at = text_place(state, me, total);
        if (lane == 0) {
            place = at;
            if (me == nb - 1) state[nb] = at == BAD ? ~0ull : at + total;
        }
    }
    __syncthreads();
    if (place == BAD) return;
    // block text -> global: bytes up to a 4-byte boundary, words, then the tail
    const uint64_t dst = place;
    const uint32_t head = (uint32_t)((4u - (uint32_t)(dst & 3u)) & 3u);
    const uint32_t h = head < total ? head : total;
    if (threadIdx.x < h) text[dst + threadIdx.x] = stage[threadIdx.x];
    const uint32_t words = (total - h) >> 2;
    uint32_t* tw = reinterpret_cast<uint32_t*>(text + dst + h);
    const uint32_t* sw = reinterpret_cast<const uint32_t*>(stage);
    for (uint32_t k = threadIdx.x; k < words; k += LINES)
        tw[k] = h == 0 ? sw[k] : __funnelshift_r(sw[k], sw[k + 1], 8u * h);
    const uint32_t t0 = h + 4u * words;
    if (threadIdx.x < total - t0) text[dst + t0 + threadIdx.x] = stage[t0 + threadIdx.x];
}

int64_t max_line(int kind) { return kind == LBM_VTK_VECTOR ? MAXLINE : 13; }

// Queues the formatting of one field: text[0..total) on the device, total in
// state[nb] (all ones if a wait inside ran out).  ticket: one uint32; state: nb + 1
// uint64, the blocks' lengths.
cudaError_t launch_format(int kind, const float* a, const float* b, const float* c, int64_t n, uint32_t* ticket,
                          uint64_t* state, char* text, cudaStream_t st) {
    const int64_t nb = (n + LINES - 1) / LINES;
    cudaError_t e = cudaMemsetAsync(ticket, 0, sizeof(uint32_t), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(state, 0, sizeof(uint64_t) * (size_t)(nb + 1), st);
    if (e != cudaSuccess || nb == 0) return e;
    switch (kind) {
        case LBM_VTK_SCALAR: vtk_emit<LBM_VTK_SCALAR><<<(unsigned)nb, LINES, 0, st>>>(a, b, c, n, ticket, state, nb, text); break;
        case LBM_VTK_SPEED: vtk_emit<LBM_VTK_SPEED><<<(unsigned)nb, LINES, 0, st>>>(a, b, c, n, ticket, state, nb, text); break;
        default: vtk_emit<LBM_VTK_VECTOR><<<(unsigned)nb, LINES, 0, st>>>(a, b, c, n, ticket, state, nb, text); break;
    }
    return cudaGetLastError();
}

std::string header(int kind, int nx, int ny, int nz) {
    const uint64_t N = (uint64_t)nx * (uint64_t)ny * (uint64_t)nz;
    std::string h = "# vtk DataFile Version 3.0\n";
    h += kind == LBM_VTK_VECTOR ? "vector" : "scalar";
    h += "\nASCII\nDATASET STRUCTURED_POINTS\nDIMENSIONS " + std::to_string(nx) + " " + std::to_string(ny) + " " +
         std::to_string(nz) + "\nORIGIN 0 0 0\nSPACING 1 1 1\nPOINT_DATA " + std::to_string(N) + "\n";
    h += kind == LBM_VTK_VECTOR ? "VECTORS vec float\n" : "SCALARS s float 1\nLOOKUP_TABLE default\n";
    return h;
}

}  // namespace vtk

// One field to one file, synchronously on the legacy default stream (ordered
// after the blocking streams that produced the field, as the reference's
// cudaMemcpy is): format on the device, copy the text back, write it.
int write_vtk_file(int kind, const float* a, const float* b, const float* c, int nx, int ny, int nz,
                   const char* path) {
    const int64_t n = (int64_t)nx * ny * nz;
    const int64_t cap = lbm_vtk_text_bound(kind, n);
    char* d_text = nullptr;
    if (cudaMalloc((void**)&d_text, (size_t)cap) != cudaSuccess) {
        set_error("write_vtk: device allocation failed");
        return LBM_ERR_ALLOC;
    }
    int64_t len = 0;
    int rc = lbm_vtk_format(kind, a, b, c, n, d_text, cap, &len, nullptr);
    std::vector<char> h;
    if (rc == LBM_OK) {
        h.resize((size_t)len);
        if (len > 0 && cudaMemcpy(h.data(), d_text, (size_t)len, cudaMemcpyDeviceToHost) != cudaSuccess) {
            set_error("write_vtk: device copy failed");
            rc = LBM_ERR_CUDA;
        }
    }
    cudaFree(d_text);
    if (rc != LBM_OK) return rc;
    FILE* f = std::fopen(path, "wb");
    if (!f) { set_error(std::string("failed to open VTK file: ") + path); return LBM_ERR_IO; }
    const std::string hd = vtk::header(kind, nx, ny, nz);
    bool ok = std::fwrite(hd.data(), 1, hd.size(), f) == hd.size();
    ok = ok && std::fwrite(h.data(), 1, h.size(), f) == h.size();
    ok = (std::fclose(f) == 0) && ok;
    if (!ok) { set_error(std::string("failed to write VTK file: ") + path); return LBM_ERR_IO; }
    return LBM_OK;
}

}  // namespace lbm

using namespace lbm::vtk;

// ---- asynchronous writer -------------------------------------------------

struct lbm_vtk_writer {
    struct Slot {
        char* d_text = nullptr;
        uint32_t* d_ticket = nullptr;
        uint64_t* d_state = nullptr;
        cudaEvent_t formatted = nullptr;
        bool busy = false;
    };
    struct Job {
        int slot;
        int kind;
        std::string path;
    };
    int nx = 0, ny = 0, nz = 0, device = 0;
    int64_t n = 0, cap = 0, nb = 0;
    size_t chunk = 0;
    char* h_text = nullptr;          // pinned, two halves of `chunk` bytes (one writer thread)
    uint64_t* h_total = nullptr;     // pinned
    std::vector<Slot> slots;
    cudaStream_t copy = nullptr;
    cudaEvent_t chunk_ev[2] = {nullptr, nullptr};
    std::mutex mu;
    std::condition_variable cv;
    std::deque<Job> jobs;
    bool stop = false;
    int error = LBM_OK;
    std::string error_msg;
    uint64_t bytes_written = 0;
    std::thread th;

    void fail(int code, const std::string& msg) {
        std::lock_guard<std::mutex> g(mu);
        if (error == LBM_OK) { error = code; error_msg = msg; }
    }

    void write_job(const Job& j) {
        Slot& s = slots[j.slot];
        if (cudaEventSynchronize(s.formatted) != cudaSuccess ||
            cudaMemcpyAsync(h_total, s.d_state + nb, sizeof(uint64_t), cudaMemcpyDeviceToHost, copy) != cudaSuccess ||
            cudaStreamSynchronize(copy) != cudaSuccess) {
            fail(LBM_ERR_CUDA, "vtk writer: formatting or copy failed");
            return;
        }
        const uint64_t total = *h_total;
        if (total > (uint64_t)cap) { fail(LBM_ERR_TIMEOUT, "vtk writer: a wait in the formatting kernel ran out"); return; }
        FILE* f = std::fopen(j.path.c_str(), "wb");
        if (!f) { fail(LBM_ERR_IO, "failed to open VTK file: " + j.path); return; }
        const std::string h = header(j.kind, nx, ny, nz);
        bool ok = std::fwrite(h.data(), 1, h.size(), f) == h.size();
        // chunks through two pinned halves: copy k + 1 while k is written
        const uint64_t nch = (total + chunk - 1) / chunk;
        auto issue = [&](uint64_t k) {
            const uint64_t o = k * chunk, len = total - o < chunk ? total - o : chunk;
            cudaMemcpyAsync(h_text + (k & 1) * chunk, s.d_text + o, len, cudaMemcpyDeviceToHost, copy);
            cudaEventRecord(chunk_ev[k & 1], copy);
        };
        if (nch > 0) issue(0);
        for (uint64_t k = 0; k < nch && ok; ++k) {
            if (k + 1 < nch) issue(k + 1);
            if (cudaEventSynchronize(chunk_ev[k & 1]) != cudaSuccess) { ok = false; break; }
            const uint64_t o = k * chunk, len = total - o < chunk ? total - o : chunk;
            ok = std::fwrite(h_text + (k & 1) * chunk, 1, len, f) == len;
            // the half just written is reused by the copy after next: issued
            // only after this fwrite, in stream order behind copy k + 1
        }
        cudaStreamSynchronize(copy);
        ok = (std::fclose(f) == 0) && ok;
        if (!ok) fail(LBM_ERR_IO, "failed to write VTK file: " + j.path);
        else {
            std::lock_guard<std::mutex> g(mu);
            bytes_written += h.size() + total;
        }
    }

    void run() {
        cudaSetDevice(device);
        for (;;) {
            Job j;
            {
                std::unique_lock<std::mutex> g(mu);
                cv.wait(g, [&] { return stop || !jobs.empty(); });
                if (jobs.empty()) return;
                j = jobs.front();
            }
            write_job(j);
            {
                std::lock_guard<std::mutex> g(mu);
                jobs.pop_front();
                slots[j.slot].busy = false;
            }
            cv.notify_all();
        }
    }
};

extern "C" {

int lbm_vtk_writer_create(int32_t nx, int32_t ny, int32_t nz, int32_t depth, lbm_vtk_writer** out) {
    if (!out || nx <= 0 || ny <= 0 || nz <= 0) { lbm::set_error("lbm_vtk_writer_create: bad argument"); return LBM_ERR_INVALID; }
    auto* w = new lbm_vtk_writer();
    w->nx = nx; w->ny = ny; w->nz = nz;
    w->n = (int64_t)nx * ny * nz;
    w->nb = (w->n + LINES - 1) / LINES;
    w->cap = w->n * max_line(LBM_VTK_VECTOR);
    w->chunk = (size_t)std::min<int64_t>(w->cap > 0 ? w->cap : 1, (int64_t)32 << 20);
    cudaGetDevice(&w->device);
    bool ok = cudaStreamCreateWithFlags(&w->copy, cudaStreamNonBlocking) == cudaSuccess &&
              cudaEventCreateWithFlags(&w->chunk_ev[0], cudaEventDisableTiming) == cudaSuccess &&
              cudaEventCreateWithFlags(&w->chunk_ev[1], cudaEventDisableTiming) == cudaSuccess &&
              cudaHostAlloc((void**)&w->h_text, 2 * w->chunk, cudaHostAllocDefault) == cudaSuccess &&
              cudaHostAlloc((void**)&w->h_total, sizeof(uint64_t), cudaHostAllocDefault) == cudaSuccess;
    w->slots.resize((size_t)(depth < 1 ? 1 : depth));
    for (auto& s : w->slots) {
        ok = ok && cudaMalloc((void**)&s.d_text, (size_t)w->cap + 16) == cudaSuccess &&
             cudaMalloc((void**)&s.d_ticket, sizeof(uint32_t)) == cudaSuccess &&
             cudaMalloc((void**)&s.d_state, sizeof(uint64_t) * (size_t)(w->nb + 1)) == cudaSuccess &&
             cudaEventCreateWithFlags(&s.formatted, cudaEventDisableTiming) == cudaSuccess;
    }
    if (!ok) {
        lbm_vtk_writer_destroy(w);
        lbm::set_error("lbm_vtk_writer_create: allocation failed");
        return LBM_ERR_ALLOC;
    }
    w->th = std::thread([w] { w->run(); });
    *out = w;
    return LBM_OK;
}

int lbm_vtk_writer_submit(lbm_vtk_writer* w, int32_t kind, const float* d_a, const float* d_b, const float* d_c,
                          const char* path, void* stream) {
    if (!w || !path || !d_a || kind < LBM_VTK_SCALAR || kind > LBM_VTK_VECTOR ||
        (kind != LBM_VTK_SCALAR && (!d_b || !d_c))) {
        lbm::set_error("lbm_vtk_writer_submit: bad argument");
        return LBM_ERR_INVALID;
    }
    int slot = -1;
    {
        std::unique_lock<std::mutex> g(w->mu);
        w->cv.wait(g, [&] {
            for (size_t k = 0; k < w->slots.size(); ++k)
                if (!w->slots[k].busy) { slot = (int)k; return true; }
            return false;
        });
        w->slots[slot].busy = true;
    }
    auto& s = w->slots[slot];
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (launch_format(kind, d_a, d_b, d_c, w->n, s.d_ticket, s.d_state, s.d_text, st) != cudaSuccess ||
        cudaEventRecord(s.formatted, st) != cudaSuccess) {
        std::lock_guard<std::mutex> g(w->mu);
        s.busy = false;
        lbm::set_error("lbm_vtk_writer_submit: launch failed");
        return LBM_ERR_CUDA;
    }
    {
        std::lock_guard<std::mutex> g(w->mu);
        w->jobs.push_back({slot, kind, path});
    }
    w->cv.notify_all();
    return LBM_OK;
}

int lbm_vtk_writer_flush(lbm_vtk_writer* w) {
    if (!w) { lbm::set_error("lbm_vtk_writer_flush: null writer"); return LBM_ERR_INVALID; }
    std::unique_lock<std::mutex> g(w->mu);
    w->cv.wait(g, [&] { return w->jobs.empty(); });
    const int e = w->error;
    if (e != LBM_OK) {
        lbm::set_error(w->error_msg);
        w->error = LBM_OK;
        w->error_msg.clear();
    }
    return e;
}

int lbm_vtk_writer_bytes(lbm_vtk_writer* w, uint64_t* bytes) {
    if (!w || !bytes) { lbm::set_error("lbm_vtk_writer_bytes: bad argument"); return LBM_ERR_INVALID; }
    std::lock_guard<std::mutex> g(w->mu);
    *bytes = w->bytes_written;
    return LBM_OK;
}

int lbm_vtk_writer_destroy(lbm_vtk_writer* w) {
    if (!w) return LBM_OK;
    if (w->th.joinable()) {
        {
            std::lock_guard<std::mutex> g(w->mu);
            w->stop = true;
        }
        w->cv.notify_all();
        w->th.join();
    }
    for (auto& s : w->slots) {
        cudaFree(s.d_text); cudaFree(s.d_ticket); cudaFree(s.d_state);
        if (s.formatted) cudaEventDestroy(s.formatted);
    }
    if (w->h_text) cudaFreeHost(w->h_text);
    if (w->h_total) cudaFreeHost(w->h_total);
    if (w->chunk_ev[0]) cudaEventDestroy(w->chunk_ev[0]);
    if (w->chunk_ev[1]) cudaEventDestroy(w->chunk_ev[1]);
    if (w->copy) cudaStreamDestroy(w->copy);
    const int e = w->error;
    delete w;
    return e;
}

int lbm_vtk_format(int32_t kind, const float* d_a, const float* d_b, const float* d_c, int64_t n, char* d_text,
                   int64_t cap, int64_t* len, void* stream) {
    if (!d_text || !len || n < 0 || kind < LBM_VTK_SCALAR || kind > LBM_VTK_VECTOR ||
        (n > 0 && (!d_a || (kind != LBM_VTK_SCALAR && (!d_b || !d_c))))) {
        lbm::set_error("lbm_vtk_format: bad argument");
        return LBM_ERR_INVALID;
    }
    if (cap < lbm_vtk_text_bound(kind, n)) { lbm::set_error("lbm_vtk_format: text buffer too small"); return LBM_ERR_INVALID; }
    const int64_t nb = (n + LINES - 1) / LINES;
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    uint64_t* scratch = nullptr;      // the blocks' lengths, the total, the ticket
    if (lbm::scratch_alloc((void**)&scratch, sizeof(uint64_t) * (size_t)(nb + 2), st) != cudaSuccess) {
        lbm::set_error("lbm_vtk_format: allocation failed");
        return LBM_ERR_ALLOC;
    }
    uint64_t total = 0;
    const bool ok = launch_format(kind, d_a, d_b, d_c, n, reinterpret_cast<uint32_t*>(scratch + nb + 1), scratch, d_text,
                                  st) == cudaSuccess &&
                    cudaMemcpyAsync(&total, scratch + nb, sizeof(uint64_t), cudaMemcpyDeviceToHost, st) == cudaSuccess;
    cudaFreeAsync(scratch, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) { lbm::set_error("lbm_vtk_format: kernel failed"); return LBM_ERR_CUDA; }
    if (!ok) { lbm::set_error("lbm_vtk_format: kernel failed"); return LBM_ERR_CUDA; }
    if (total > (uint64_t)cap) { lbm::set_error("lbm_vtk_format: a wait in the kernel ran out"); return LBM_ERR_TIMEOUT; }
    *len = (int64_t)total;
    return LBM_OK;
}

int64_t lbm_vtk_text_bound(int32_t kind, int64_t n) { return n * max_line(kind) + 16; }

int lbm_format_g6(const float* v, int64_t n, char* out, int32_t stride, uint8_t* lens) {
    if ((!v || !out || !lens) && n > 0) { lbm::set_error("lbm_format_g6: null argument"); return LBM_ERR_INVALID; }
    if (stride < 12) { lbm::set_error("lbm_format_g6: stride below 12"); return LBM_ERR_INVALID; }
    for (int64_t i = 0; i < n; ++i) lens[i] = (uint8_t)fmt_g6(v[i], out + i * stride);
    return LBM_OK;
}

}  // extern "C"
