// Generator of loop-fused elementwise / reduction / row kernels for sm_100a.
//
// One fusion body (elementwise prims, layout prims, gathers, and reductions over the trailing axis) becomes ONE
// kernel over a [R, C] iteration space: a group of T threads walks each row in 16-byte vector chunks, reductions
// over the row are combined with warp shuffles (and shared memory across warps), and everything that reads a
// reduction result is recomputed from registers in a later phase over the same row, so each input element is
// read from HBM once. This is the counterpart of the reference's generated elementwise kernel
// (lumen/codegen/elementwise/cuda/mod.rs:54-333, kernel.py:56-167), of its Triton reduction kernels with fused
// prologue/epilogue (lumen/codegen/reduction/triton.rs) and of its row kernels for normalization diamonds
// (lumen/codegen/row/triton.rs), all of which only exist off-Blackwell.
//
// Numerics follow the reference interpreter (lumen/reference/mod.rs:442-695): one rounding to the result dtype
// after every primitive (16-bit floats are widened to f32, operated on once, rounded back), no multiply-add
// contraction (NVRTC --fmad=false), NaN-propagating max, integer division by zero = -1, two's complement wrap,
// saturating float->int casts, gather indices clamped. Row sums are combined in tree order, not the
// interpreter's sequential order: that is the one tolerance-level difference (reference tests allow 1e-5).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <functional>
#include <map>
#include <set>
#include <sstream>

#include "fused.h"

namespace lb {
namespace {

const char* kPreamble = R"CUDA(
typedef long long i64; typedef unsigned long long u64; typedef unsigned int u32; typedef unsigned short u16;
typedef unsigned char u8; typedef signed char i8; typedef short i16; typedef int i32;
__device__ __forceinline__ float bf16_to_f32(u16 b) { return __uint_as_float(((u32)b) << 16); }
__device__ __forceinline__ u16 f32_to_bf16(float x) { u16 r; asm("cvt.rn.bf16.f32 %0, %1;" : "=h"(r) : "f"(x)); return r; }
__device__ __forceinline__ float rnd_bf16(float x) { return bf16_to_f32(f32_to_bf16(x)); }
__device__ __forceinline__ float f16_to_f32(u16 b) { float r; asm("cvt.f32.f16 %0, %1;" : "=f"(r) : "h"(b)); return r; }
__device__ __forceinline__ u16 f32_to_f16(float x) { u16 r; asm("cvt.rn.f16.f32 %0, %1;" : "=h"(r) : "f"(x)); return r; }
__device__ __forceinline__ float rnd_f16(float x) { return f16_to_f32(f32_to_f16(x)); }
__device__ __forceinline__ float rnd_f32(float x) { return x; }
__device__ __forceinline__ double rnd_f64(double x) { return x; }
__device__ __forceinline__ float fmax_nan(float a, float b) { float r; asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b)); return r; }
// exp(x) of a softmax normaliser's term, x = value - row maximum <= 0, that is only summed: one multiply and one
// ex2.approx. Its relative error grows with |x| (to 5e-6 at -87) and results below 2^-126 flush to zero, but a term's
// weight in the sum (which holds exp(0) = 1) shrinks faster: the sum is within 2^-21 of the exactly rounded one.
__device__ __forceinline__ float exp_sum_term(float x) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__fmul_rn(x, 1.4426950408889634f))); return r; }
__device__ __forceinline__ double fmax_nan(double a, double b) { return (a != a || b != b) ? __longlong_as_double(0x7ff8000000000000LL) : fmax(a, b); }
__device__ __forceinline__ float fmin_nan(float a, float b) { float r; asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ double fmin_nan(double a, double b) { return (a != a || b != b) ? __longlong_as_double(0x7ff8000000000000LL) : fmin(a, b); }
// Zero at run time (every launch of these kernels has one block along z), unknown at compile time. Integer negations are
// written RT_ZERO - x: with CUDA 12.9 for sm_100a, a chain of three or more signed 32-bit max (or min) whose operands
// are literal negations 0 - x comes out as the extremum over x and -x together (a stand-alone kernel shows it with
// `neg.s32` in inline assembly as well, so it happens after PTX); a subtraction from a register does not.
#define RT_ZERO blockIdx.z
// Waits for the kernels before this one in the stream, which this one may have become resident before: the thread's index, and then
// the pointers through which the kernel reads, as values that come out of the wait. Every load's address is computed from one of
// those pointers, so none can be moved in front of the wait - also not the loads of read-only memory (__ldg), which a compiler may
// move across a memory clobber, where neither the thread nor the block is part of the address (a scalar, a row's own operand).
__device__ __forceinline__ u32 grid_wait() {
    u32 tid = threadIdx.x;
    asm volatile("griddepcontrol.wait;" : "+r"(tid) : : "memory");
    return tid;
}
template <class T> __device__ __forceinline__ T* behind_wait(T* p, u32 tid) {
    size_t at = __cvta_generic_to_global(p);
    asm volatile("" : "+l"(at) : "r"(tid));
    return (T*)__cvta_global_to_generic(at);  // known to lead to global memory
}
template <class T> __device__ __forceinline__ T imax(T a, T b) { return a > b ? a : b; }
template <class T> __device__ __forceinline__ T imin(T a, T b) { return a < b ? a : b; }
// division by zero gives all ones and leaves the remainder a; a signed -1 divisor negates (wrapping at the lowest
// value, where the hardware division would trap or is undefined) - an unsigned divisor of all ones is an ordinary one
template <class T, class U> __device__ __forceinline__ T idiv(T a, T b) {
    if (b == 0) return (T)-1;
    if ((T)-1 < (T)0 && b == (T)-1) return (T)((U)RT_ZERO - (U)a);
    return a / b;
}
template <class T> __device__ __forceinline__ T irem(T a, T b) {
    if (b == 0) return a;
    if ((T)-1 < (T)0 && b == (T)-1) return 0;
    return a % b;
}
// float -> integer as a cast does: saturating, NaN to 0
template <class T> __device__ __forceinline__ T sat_cast(double x, double lo, double hi, T tlo, T thi) {
    if (x != x) return (T)0;
    if (x <= lo) return tlo;
    if (x >= hi) return thi;
    return (T)x;
}
template <int BYTES> struct VecBytes;
template <> struct VecBytes<16> { typedef uint4 type; };
template <> struct VecBytes<8> { typedef uint2 type; };
template <> struct VecBytes<4> { typedef u32 type; };
template <> struct VecBytes<2> { typedef u16 type; };
template <> struct VecBytes<1> { typedef u8 type; };
// V consecutive elements of T, moved in the widest pieces up to 16 bytes
template <class T, int V> __device__ __forceinline__ void ldv(const T* __restrict__ p, T* dst) {
    constexpr int B = sizeof(T) * V; constexpr int P = B >= 16 ? 16 : B; typedef typename VecBytes<P>::type W;
    #pragma unroll
    for (int k = 0; k < B / P; k++) ((W*)dst)[k] = __ldg((const W*)p + k);
}
template <class T, int V> __device__ __forceinline__ void ldv_plain(const T* p, T* dst) {
    constexpr int B = sizeof(T) * V; constexpr int P = B >= 16 ? 16 : B; typedef typename VecBytes<P>::type W;
    #pragma unroll
    for (int k = 0; k < B / P; k++) ((W*)dst)[k] = ((const W*)p)[k];
}
template <class T, int V> __device__ __forceinline__ void stv(T* p, const T* src) {
    constexpr int B = sizeof(T) * V; constexpr int P = B >= 16 ? 16 : B; typedef typename VecBytes<P>::type W;
    #pragma unroll
    for (int k = 0; k < B / P; k++) ((W*)p)[k] = ((const W*)src)[k];
}
// The same at element `at` (a multiple of V) of an array of `total`, of which the last V may lie partly behind its end (where the last
// element stands in: a value as good as its neighbours, so that what is computed from it takes no path of its own)
template <class T, int V, class I> __device__ __forceinline__ void ldv_within(const T* __restrict__ p, I at, I total, T* dst) {
    if (at + V <= total) { ldv<T, V>(p + at, dst); return; }
    #pragma unroll
    for (int k = 0; k < V; k++) dst[k] = __ldg(p + (at + k < total ? at + k : total - 1));
}
template <class T, int V, class I> __device__ __forceinline__ void ldv_within_plain(const T* p, I at, I total, T* dst) {
    if (at + V <= total) { ldv_plain<T, V>(p + at, dst); return; }
    #pragma unroll
    for (int k = 0; k < V; k++) dst[k] = p[at + k < total ? at + k : total - 1];
}
// Elements [at - shift, at - shift + V) of an array of `total`, 0 <= shift < V, at a multiple of V: two aligned pieces, whose bytes are
// moved by the shift (the same for every thread). Others of the array's elements stand in before the first and behind the last.
template <class T, int V, class I> __device__ __forceinline__ void ldv_shifted(const T* __restrict__ p, I at, int shift, I total, T* dst) {
    constexpr int B = sizeof(T) * V;
    if constexpr (B != 16 || sizeof(T) > 4 || sizeof(T) < 2) {
        #pragma unroll
        for (int k = 0; k < V; k++) { const I i = at - shift + k; dst[k] = __ldg(p + (i < 0 ? 0 : i < total ? i : total - 1)); }
    } else {
        __align__(16) u32 w[8];
        ldv_within<T, V, I>(p, at >= V ? at - V : at, total, (T*)w);
        ldv_within<T, V, I>(p, at, total, (T*)(w + 4));
        const int from = B - shift * (int)sizeof(T);  // first byte, in (0, 16]
        #pragma unroll
        for (int k = 0; k < 8; k++) w[k] = from & 16 ? w[k < 4 ? k + 4 : k] : w[k];
        #pragma unroll
        for (int k = 0; k < 6; k++) w[k] = from & 8 ? w[k + 2] : w[k];
        #pragma unroll
        for (int k = 0; k < 5; k++) w[k] = from & 4 ? w[k + 1] : w[k];
        if (sizeof(T) == 2) {
            #pragma unroll
            for (int k = 0; k < 4; k++) w[k] = from & 2 ? __funnelshift_r(w[k], w[k + 1], 16) : w[k];
        }
        #pragma unroll
        for (int k = 0; k < 4; k++) ((u32*)dst)[k] = w[k];
    }
}
// Stores those of V consecutive elements that lie in [0, cols), the first of them at column c of the row at p
template <class T, int V, class I> __device__ __forceinline__ void stv_within(T* p, I c, I cols, const T* src) {
    if (c >= 0 && c + V <= cols) { stv<T, V>(p + c, src); return; }
    if constexpr (V > 1) {
        stv_within<T, V / 2, I>(p, c, cols, src);
        stv_within<T, V / 2, I>(p, c + V / 2, cols, src + V / 2);
    }
}
template <class T> __device__ __forceinline__ T shfl_xor_any(T v, int m) {
    if (sizeof(T) == 8) { u64 b; memcpy(&b, &v, 8); b = __shfl_xor_sync(0xffffffffu, b, m); memcpy(&v, &b, 8); return v; }
    u32 b = 0; memcpy(&b, &v, sizeof(T)); b = __shfl_xor_sync(0xffffffffu, b, m); memcpy(&v, &b, sizeof(T)); return v;
}

// ---- two elements per step ("pair mode"): p2<T> holds lanes e and e+1; bfloat16 pairs stay packed in one register and
// use the native packed instructions (one rounding of the exact result per lane, as the reference interpreter rounds) ----
template <class T> struct p2 { T x, y; };
struct bf16x2 { u32 v; };
template <class T> __device__ __forceinline__ T L0(T s) { return s; }
template <class T> __device__ __forceinline__ T L1(T s) { return s; }
template <class T> __device__ __forceinline__ T L0(p2<T> v) { return v.x; }
template <class T> __device__ __forceinline__ T L1(p2<T> v) { return v.y; }
__device__ __forceinline__ float L0(bf16x2 v) { return __uint_as_float(v.v << 16); }
__device__ __forceinline__ float L1(bf16x2 v) { return __uint_as_float(v.v & 0xffff0000u); }
// rounds two floats to bfloat16 (nearest even) with one conversion; lane 0 in the low half
__device__ __forceinline__ bf16x2 mk_bf16x2(float lo, float hi) { bf16x2 r; asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r.v) : "f"(hi), "f"(lo)); return r; }
// packs two floats that already are bfloat16 values (no rounding)
__device__ __forceinline__ bf16x2 pk_bf16x2(float lo, float hi) { bf16x2 r; r.v = (__float_as_uint(lo) >> 16) | (__float_as_uint(hi) & 0xffff0000u); return r; }
__device__ __forceinline__ bf16x2 to_bf16x2(bf16x2 v) { return v; }
__device__ __forceinline__ bf16x2 to_bf16x2(float s) { bf16x2 r; r.v = (__float_as_uint(s) >> 16) * 0x10001u; return r; }
__device__ __forceinline__ bf16x2 ld_bf16x2(const u16* p) { bf16x2 r; r.v = *(const u32*)p; return r; }
__device__ __forceinline__ bf16x2 bf16x2_add(bf16x2 a, bf16x2 b) { bf16x2 r; asm("add.rn.bf16x2 %0, %1, %2;" : "=r"(r.v) : "r"(a.v), "r"(b.v)); return r; }
__device__ __forceinline__ bf16x2 bf16x2_sub(bf16x2 a, bf16x2 b) { bf16x2 r; asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(r.v) : "r"(a.v), "r"(b.v)); return r; }
__device__ __forceinline__ bf16x2 bf16x2_mul(bf16x2 a, bf16x2 b) { bf16x2 r; asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r.v) : "r"(a.v), "r"(b.v)); return r; }
__device__ __forceinline__ bf16x2 bf16x2_max(bf16x2 a, bf16x2 b) { bf16x2 r; asm("max.NaN.bf16x2 %0, %1, %2;" : "=r"(r.v) : "r"(a.v), "r"(b.v)); return r; }
__device__ __forceinline__ bf16x2 bf16x2_min(bf16x2 a, bf16x2 b) { bf16x2 r; asm("min.NaN.bf16x2 %0, %1, %2;" : "=r"(r.v) : "r"(a.v), "r"(b.v)); return r; }
__device__ __forceinline__ bf16x2 bf16x2_neg(bf16x2 a) { bf16x2 r; r.v = a.v ^ 0x80008000u; return r; }
__device__ __forceinline__ bf16x2 bf16x2_abs(bf16x2 a) { bf16x2 r; r.v = a.v & 0x7fff7fffu; return r; }
// float32 pairs: the packed add / mul / fma of sm_100, one rounding per lane exactly as the scalar instructions
__device__ __forceinline__ p2<float> to_f32x2(p2<float> v) { return v; }
__device__ __forceinline__ p2<float> to_f32x2(float s) { p2<float> r = {s, s}; return r; }
__device__ __forceinline__ p2<float> f32x2_add(p2<float> a, p2<float> b) {
    p2<float> r;
    asm("{\n\t.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tadd.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ p2<float> f32x2_mul(p2<float> a, p2<float> b) {
    p2<float> r;
    asm("{\n\t.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmul.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
// a - b as fma(b, -1, a): exact product, one rounding of the difference
__device__ __forceinline__ p2<float> f32x2_sub(p2<float> a, p2<float> b) {
    p2<float> r;
    asm("{\n\t.reg .b64 ra, rb, rm, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rm, {%6, %6};\n\tfma.rn.f32x2 rd, rb, rm, ra;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(-1.0f));
    return r;
}
__device__ __forceinline__ p2<float> f32x2_fma(p2<float> a, p2<float> b, p2<float> c) {
    p2<float> r;
    asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%6, %7};\n\tfma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return r;
}
// Division of a chunk's elements by one divisor, the correctly rounded quotients as __fdiv_rn gives them: with y = RN(1 / b),
// q0 = RN(a y), q1 = RN(q0 + (a - b q0) y) is within an ulp and q2 = RN(q1 + (a - b q1) y) is RN(a / b) (Markstein, "Computation
// of elementary functions on the IBM RISC System/6000 processor", 1990, theorem 5.1: y correctly rounded, the residual exact). That holds
// where nothing under- or overflows: 2^-40 <= b <= 2^40 and 2^-60 <= |a| <= 2^60 for every a that is not zero (which
// is its own quotient); what is outside is divided as usual. 2.5 packed instructions an element in one block of
// straight-line code, where a division each is ten and a branch that nothing is scheduled across, and a zero leaves even that one: a layer norm
// of 8192 x 1024 bfloat16 with its gradients, which takes three quotients an element and is bound by its instructions, 33.4 -> 28.3 us;
// relu(x) over its row's sum, 32768 x 1024, float32 67.8 -> 44.4, bfloat16 65.7 -> 34.1; a layer norm of as many elements with every other row
// zero 63.3 -> 46.2, 54.3 -> 33.6. 3.2e9 random quotients equal __fdiv_rn's. Divided as usual, elements cost more than where they are from the
// start (float32 softmax of logits that spread by 80: 64 us against 50): may_be_tiny keeps away those that often are.
#define LEAST_DIVIDEND 8.673617379884035e-19f
#define MOST_DIVIDEND 1.152921504606847e18f
__device__ __forceinline__ float row_reciprocal(float b) { return b >= 9.094947017729282e-13f && b <= 1.099511627776e12f ? __frcp_rn(b) : 0.0f; }
__device__ __forceinline__ void abs_range(p2<float> a, float& lo, float& hi) {
    lo = fminf(lo, fminf(fabsf(a.x), fabsf(a.y))), hi = fmaxf(hi, fmaxf(fabsf(a.x), fabsf(a.y)));
}
__device__ __forceinline__ void abs_range(float a, float& lo, float& hi) { lo = fminf(lo, fabsf(a)), hi = fmaxf(hi, fabsf(a)); }
__device__ __forceinline__ p2<float> quotient(p2<float> a, float b, float y) {
    const p2<float> mb = {-b, -b}, yy = {y, y};
    p2<float> q = f32x2_mul(a, yy);
    q = f32x2_fma(f32x2_fma(mb, q, a), yy, q);
    return f32x2_fma(f32x2_fma(mb, q, a), yy, q);
}
__device__ __forceinline__ float quotient(float a, float b, float y) {
    float q = __fmul_rn(a, y);
    q = __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
    return __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
}
// Four elements of a chunk that holds zeros or what is outside the range. Not inlined: such code between that of the other chunks costs
// those, the layer norm above 28.3 -> 29.8 us.
__device__ __noinline__ float4 quotients_any(float4 a, float b, float y) {
    float lo = 1.0f, hi = 1.0f;
    abs_range(a.x == 0.0f ? 1.0f : a.x, lo, hi), abs_range(a.y == 0.0f ? 1.0f : a.y, lo, hi);
    abs_range(a.z == 0.0f ? 1.0f : a.z, lo, hi), abs_range(a.w == 0.0f ? 1.0f : a.w, lo, hi);
    if (y != 0.0f && lo >= LEAST_DIVIDEND && hi <= MOST_DIVIDEND)  // (b > 0: a zero is its own quotient)
        return make_float4(a.x == 0.0f ? a.x : quotient(a.x, b, y), a.y == 0.0f ? a.y : quotient(a.y, b, y), a.z == 0.0f ? a.z : quotient(a.z, b, y),
                           a.w == 0.0f ? a.w : quotient(a.w, b, y));
    return make_float4(__fdiv_rn(a.x, b), __fdiv_rn(a.y, b), __fdiv_rn(a.z, b), __fdiv_rn(a.w, b));
}
__device__ __forceinline__ void divide_any(const p2<float>* a, p2<float>* q, float b, float y) {
    const float4 r = quotients_any(make_float4(a[0].x, a[0].y, a[1].x, a[1].y), b, y);
    q[0].x = r.x, q[0].y = r.y, q[1].x = r.z, q[1].y = r.w;
}
__device__ __forceinline__ void divide_any(const float* a, float* q, float b, float y) {
    const float4 r = quotients_any(make_float4(a[0], a[1], a[2], a[3]), b, y);
    q[0] = r.x, q[1] = r.y, q[2] = r.z, q[3] = r.w;
}
// What the magnitudes of a chunk's elements lie between. Divided, it becomes the quotients' range, or one that nothing is taken to fit.
struct Magnitudes { float least, most; };
template <int N, class T> __device__ __forceinline__ void divide_within(const T* a, T* q, float b, float y, Magnitudes& range) {
    if (y != 0.0f && range.least >= LEAST_DIVIDEND && range.most <= MOST_DIVIDEND) {
        #pragma unroll
        for (int k = 0; k < N; k++) q[k] = quotient(a[k], b, y);
        range.least *= y * 0.999f, range.most *= y * 1.001f;
    } else {
        #pragma unroll
        for (int k = 0; k < N; k += 16 / (int)sizeof(T)) divide_any(a + k, q + k, b, y);
        range.least = 0.0f;
    }
}
template <int N, class T> __device__ __forceinline__ Magnitudes divide_chunk(const T* a, T* q, float b, float y) {
    Magnitudes range = {1.0f, 1.0f};
    #pragma unroll
    for (int k = 0; k < N; k++) abs_range(a[k], range.least, range.most);
    divide_within<N>(a, q, b, y, range);
    return range;
}
// A chunk of quotients by `b`, which lie in `range`, divided by it again: the elements are not looked over a second time.
template <int N, class T> __device__ __forceinline__ Magnitudes divide_again(const T* a, T* q, float b, float y, Magnitudes range) {
    divide_within<N>(a, q, b, y, range);
    return range;
}
)CUDA";

struct CType {
    const char* compute;  // type values are computed in
    const char* memory;   // type stored in global memory
    const char* unsigned_t;
};

CType ctype(int dtype) {
    switch (dtype) {
        case LB_BOOL: return {"bool", "u8", "u8"};
        case LB_I8: return {"i8", "i8", "u8"};
        case LB_I16: return {"i16", "i16", "u16"};
        case LB_I32: return {"i32", "i32", "u32"};
        case LB_I64: return {"i64", "i64", "u64"};
        case LB_U8: return {"u8", "u8", "u8"};
        case LB_U16: return {"u16", "u16", "u16"};
        case LB_U32: return {"u32", "u32", "u32"};
        case LB_U64: return {"u64", "u64", "u64"};
        case LB_F16: return {"float", "u16", ""};
        case LB_BF16: return {"float", "u16", ""};
        case LB_F32: return {"float", "float", ""};
        case LB_F64: return {"double", "double", ""};
    }
    fail(LB_ERR_INVALID, "bad dtype");
}

const char* rnd_fn(int dtype) {
    switch (dtype) {
        case LB_F16: return "rnd_f16";
        case LB_BF16: return "rnd_bf16";
        case LB_F32: return "rnd_f32";
        case LB_F64: return "rnd_f64";
    }
    return "";
}

// memory value -> compute value
std::string from_memory(int dtype, const std::string& x) {
    switch (dtype) {
        case LB_BOOL: return "(" + x + " != 0)";
        case LB_F16: return "f16_to_f32(" + x + ")";
        case LB_BF16: return "bf16_to_f32(" + x + ")";
        default: return x;
    }
}
std::string to_memory(int dtype, const std::string& x) {
    switch (dtype) {
        case LB_BOOL: return "(u8)(" + x + " ? 1 : 0)";
        case LB_F16: return "f32_to_f16(" + x + ")";
        case LB_BF16: return "(u16)(__float_as_uint(" + x + ") >> 16)";  // values are already rounded to bf16
        default: return x;
    }
}

std::string float_literal(double v, int dtype) {
    if (dtype == LB_F64) {
        uint64_t b;
        memcpy(&b, &v, 8);
        return format("__longlong_as_double(0x%llxLL)", (unsigned long long)b);
    }
    float f = (float)v;
    uint32_t b;
    memcpy(&b, &f, 4);
    return format("__uint_as_float(0x%xu)", b);
}

// round-to-nearest-even f32 -> bf16 / f16 on the host, for constants
double host_round(double x, int dtype) {
    if (dtype == LB_F64) return x;
    // single rounding through a round-to-odd f32 (lumen/tensor/dtype.rs:217-239)
    float f = (float)x;
    if (dtype == LB_F32) return f;
    uint32_t bits;
    memcpy(&bits, &f, 4);
    if (std::isfinite(f) && (double)f != x && !(bits & 1)) {
        bool outward = ((double)f < x) != std::signbit(f);
        bits = outward ? bits + 1 : bits - 1;
        memcpy(&f, &bits, 4);
    }
    if (dtype == LB_BF16) {
        if ((bits & 0x7fffffffu) > 0x7f800000u) return NAN;
        uint32_t r = 0x8000u;
        if ((bits & r) && (bits & (3 * r - 1))) bits += r;
        bits &= 0xffff0000u;
        memcpy(&f, &bits, 4);
        return f;
    }
    // f16
    if (std::isnan(f)) return NAN;
    double a = std::fabs((double)f), r;
    if (a >= 65520.0) r = INFINITY;
    else if (a < 6.103515625e-05) r = std::nearbyint(a * 16777216.0) / 16777216.0;
    else {
        int e;
        std::frexp(a, &e);
        double ulp = std::ldexp(1.0, e - 11);
        r = std::nearbyint(a / ulp) * ulp;
    }
    return std::signbit(f) ? -r : r;
}

struct Comp {
    std::string expr;  // the coordinate, may reference r, c0, e
    std::string base;  // when lane: expr == base + e, base a multiple of VEC not referencing e
    bool lane = false, e_dep = false, row_dep = false, c_dep = false;
    bool dyn = false;  // references a variable defined inside a phase (a gathered index)
    int64_t zero_known = 0;  // 1 when the coordinate is the constant 0
};
typedef std::vector<Comp> Index;

Comp zero_comp() {
    Comp c;
    c.expr = "0";
    c.zero_known = 1;
    return c;
}

struct Phase {
    std::string pre, body, post;
    std::map<std::string, std::string> memo;
    // What is done for a whole chunk at once (a division of its elements) cuts the loop over the elements: the parts before the cuts,
    // each with what follows it, and the variables of the loop by the part that defines them. `body` is the part being written.
    struct Part { std::string body, then, key, array, type; };
    std::vector<Part> parts;
    struct BodyVar { std::string type, name; size_t part; };
    std::vector<BodyVar> body_vars;
    std::string chunk_decls;  // arrays of a chunk
    // reduction phases
    bool reduces = false;
    std::string acc, acc_type, init, combine_a_b;  // combine as a format with %A %B
    int sums = 1;  // how many a thread keeps
    std::string result;
    bool chunked = true;  // false for the row epilogue (runs once per row, no column loop)
};

std::string subst(std::string s, const std::string& a, const std::string& b) {
    std::string out;
    for (size_t k = 0; k < s.size(); k++) {
        if (s[k] == '%' && k + 1 < s.size() && (s[k + 1] == 'A' || s[k + 1] == 'B')) {
            out += s[k + 1] == 'A' ? a : b;
            k++;
        } else {
            out += s[k];
        }
    }
    return out;
}

class Generator {
  public:
    Generator(const Module& module, const Graph& g) : module_(module), g_(g) {}

    FusedKernel run() {
        plan_space();
        // phases are created on demand while generating the outputs
        Phase main_phase, epilogue;
        epilogue.chunked = false;
        std::vector<std::pair<int, int>> full_outputs, row_outputs;  // (output position, value)
        for (size_t k = 0; k < g_.outputs.size(); k++) {
            const TensorType& t = g_.type(g_.outputs[k]);
            if (behind_columns_.count(g_.outputs[k])) {
                column_outputs_.push_back((int)k);
                continue;
            }
            if (t.numel() == R_ * C_ && (C_ != 1 || !has_reduce_)) full_outputs.push_back({(int)k, g_.outputs[k]});
            else if (t.numel() == R_) row_outputs.push_back({(int)k, g_.outputs[k]});
            else
                fail(LB_ERR_UNSUPPORTED, format("fusion output %s does not span the [%lld, %lld] iteration space",
                                                t.str().c_str(), (long long)R_, (long long)C_));
        }
        // Row outputs first: generating them creates the reduction phases.
        for (auto [k, v] : row_outputs) {
            const TensorType& t = g_.type(v);
            Index idx = output_index(t, false);
            std::string val = gen(v, idx, epilogue);
            epilogue.pre += format("if (active && lane_in_row == 0) ((%s*)out%d)[r] = %s;\n", ctype(t.dtype).memory, k,
                                   to_memory(t.dtype, val).c_str());
        }
        // A full output is stored by the first phase that already computes its value (a reduction's prologue),
        // so it is neither recomputed nor re-read; otherwise by a final phase over the row.
        bool main_used = false;
        for (auto [k, v] : full_outputs) {
            const TensorType& t = g_.type(v);
            Index idx = output_index(t, true);
            Phase* home = &main_phase;
            for (Phase& ph : phases_)
                if (ph.chunked && ph.memo.count(key_of(v, idx))) {
                    home = &ph;
                    break;
                }
            main_used |= home == &main_phase;
            std::string val = gen(v, idx, *home);
            CType ct = ctype(t.dtype);
            std::string buf = format("ob%d", k);
            home->pre += format("__align__(16) %s %s[VEC];\n", ct.memory, buf.c_str());
            home->body += store_element(buf, t.dtype, val);
            if (shifted_)
                home->post += format("if (active) stv_within<%s, VEC, idx_t>((%s*)out%d + r * (idx_t)NCOLS, c0, (idx_t)NCOLS, %s);\n", ct.memory, ct.memory, k, buf.c_str());
            else
                home->post += format("if (active) stv<%s, VEC>((%s*)out%d + (r * (idx_t)NCOLS + c0), %s);\n", ct.memory,
                                     ct.memory, k, buf.c_str());
        }
        // Column sums: a thread keeps its columns for all the rows its CTA walks, so the partial sums stay in registers.
        for (size_t k = 0; k < col_reduces_.size(); k++) {
            const Node& n = *g_.node_of(col_reduces_[k]);
            Index idx = column_operand_index(g_.type(n.inputs[0]), n.ints("axes").size());
            Phase* home = &main_phase;
            for (Phase& ph : phases_)
                if (ph.chunked && ph.memo.count(key_of(n.inputs[0], idx))) {
                    home = &ph;
                    break;
                }
            main_used |= home == &main_phase;
            std::string val = gen(n.inputs[0], idx, *home), init, combine;
            reduce_ops(n, g_.type(n.output), &init, &combine);
            home->body += "if (active) {\n" + accumulate(format("cacc%d[ch][e]", (int)k), combine, val) + "}\n";
        }
        if (main_used) phases_.push_back(main_phase);
        if (!row_outputs.empty()) phases_.push_back(epilogue);
        return emit();
    }

  private:
    const Module& module_;
    const Graph& g_;
    int64_t R_ = 1, C_ = 1;
    int VEC_ = 1, T_ = 1, RPB_ = 1, NCH_ = 1;
    bool has_reduce_ = false;
    bool wide_index_ = false;
    int counter_ = 0;
    std::vector<Phase> phases_;
    std::map<std::string, std::string> reduce_memo_;
    std::string row_decls_;     // row-scope declarations (reduction results)
    std::string kernel_cache_;  // CTA-scope cached column loads
    std::string row_cache_;     // row-scope cached loads
    struct RowCache { std::string type, buf, load; int bytes; };
    std::vector<RowCache> row_caches_;  // the same loads one by one, for prefetching the next row block
    std::map<std::string, std::string> cached_loads_;
    int cached_regs_ = 0;

    // Row and column reductions in one kernel: the values read from column totals (generated in fused_finalize), and the
    // outputs among them by position.
    std::set<int> behind_columns_;
    std::vector<int> column_outputs_;
    int resident_ = 1;  // CTAs per SM a kernel with column sums is built for and launched with
    bool sixteen_warps_ = false;  // no kernel of row and column sums has more on an SM, and more slices than it once had
    bool shifts_ = true, shifted_ = false;  // may start, starts a row's chunks at aligned addresses before its first element
    bool narrow_ = false;                   // 16-bit tensors
    int period_ = 1;                        // ... rows that far apart at the same distance

    std::string fresh(const char* prefix) { return format("%s%d", prefix, counter_++); }

    // ---- iteration space ----------------------------------------------------------------------------------
    void plan_space() {
        const TensorType* space = nullptr;
        int64_t col_r = -1, col_c = -1;
        for (const Node& n : g_.nodes) {
            for (int v : n.inputs)
                if (behind_columns_.count(v)) behind_columns_.insert(n.output);
            if (n.op != "reduce_sum" && n.op != "reduce_max") continue;
            const TensorType& x = g_.type(n.inputs[0]);
            auto axes = n.ints("axes");
            std::sort(axes.begin(), axes.end());
            int lead = 0;
            if (mixed_ && leading_axes(n, x, &lead)) {
                int64_t r = 1;
                for (int d = 0; d < lead; d++) r *= x.shape[d];
                const int64_t c = r ? x.numel() / r : 0;
                if (!r || !c || (col_r >= 0 && (r != col_r || c != col_c)) || behind_columns_.count(n.inputs[0]))
                    fail(LB_ERR_UNSUPPORTED, "column reductions over different shapes in one fusion");
                col_r = r, col_c = c;
                col_reduces_.push_back(n.output);
                behind_columns_.insert(n.output);
                continue;
            }
            if (behind_columns_.count(n.inputs[0])) fail(LB_ERR_UNSUPPORTED, "a row reduction of column totals in one fusion");
            for (size_t k = 0; k < axes.size(); k++)
                if (axes[k] != (int64_t)(x.rank() - axes.size() + k))
                    fail(LB_ERR_UNSUPPORTED,
                         format("%s over axes other than the trailing ones of %s has no fused row kernel", n.op.c_str(),
                                x.str().c_str()));
            int64_t c = 1;
            for (auto a : axes) c *= x.shape[a];
            int64_t r = x.numel() / std::max<int64_t>(c, 1);
            if (has_reduce_ && (c != C_ || r != R_))
                fail(LB_ERR_UNSUPPORTED, "reductions over different row shapes in one fusion");
            has_reduce_ = true;
            C_ = c;
            R_ = c ? r : 0;
            space = &x;
        }
        if (mixed_) {
            if (has_reduce_ && (R_ != col_r || C_ != col_c)) fail(LB_ERR_UNSUPPORTED, "row and column reductions over different shapes in one fusion");
            R_ = col_r, C_ = col_c, has_reduce_ = true;
        } else if (!has_reduce_) {
            for (int v : g_.outputs)
                if (!space || g_.type(v).numel() > space->numel()) space = &g_.type(v);
            if (!space) fail(LB_ERR_INVALID, "fusion without outputs");
            // A pure elementwise space is flat: the row is the last dimension, widened by a divisor of the
            // leading dimensions until it is long enough to keep a thread group busy.
            C_ = space->rank() ? space->shape.back() : 1;
            // (the horizontal form keeps the last dimension as its row: every group's size is a multiple of it)
            const int64_t longest = 64LL * 1024 * 4;  // what one block takes as a row (64 chunks of 1024 threads x 4 elements)
            for (int d = space->rank() - 2; !multi_ && d >= 0 && C_ > 0 && C_ < 1024; d--) {
                int64_t n = space->shape[d], k = 1;
                while (k < n && (n % k != 0 || C_ * k < 1024)) k++;
                if (C_ * k > longest) {  // no divisor of this dimension gives a row of a good length: the largest that fits
                    for (k = std::min<int64_t>(n, 16384 / C_); k > 1 && n % k != 0;) k--;
                    C_ *= std::max<int64_t>(k, 1);
                    break;
                }
                C_ *= k;
                if (k < n) break;
            }
            if (!multi_ && C_ > longest) {  // a last dimension longer than a block's row: rows are a divisor of it
                int64_t c = 16384;
                while (c > 1 && C_ % c != 0) c--;
                C_ = c;
            }
            R_ = C_ ? space->numel() / C_ : 0;
        }
        // vector width: 16 bytes of the narrowest tensor spanning the space, dividing C
        int min_size = 8;
        auto consider = [&](const TensorType& t) {
            if (t.numel() == R_ * C_ || t.numel() == C_) min_size = std::min(min_size, dtype_size(t.dtype));
        };
        for (int v : g_.inputs) consider(g_.type(v));
        for (int v : g_.outputs) consider(g_.type(v));
        const int widest = std::min(8, 16 / min_size);
        narrow_ = min_size <= 2;
        VEC_ = widest;
        while (VEC_ > 1 && C_ % VEC_ != 0) VEC_ /= 2;
        shifted_ = VEC_ == 1 && widest == 8 && shifts_ && !mixed_ && shiftable(*space, widest);
        if (shifted_) VEC_ = widest;
        auto vectors = [&] { return std::max<int64_t>((C_ + VEC_ - 1 + (shifted_ ? VEC_ - 1 : 0)) / VEC_, 1); };
        int64_t nvec = vectors();
        const int64_t per = vectors_per_thread(nvec);
        int64_t want = (nvec + per - 1) / per;
        T_ = 1;
        while (T_ < want && T_ < 1024) T_ *= 2;
        if (shifted_ && T_ > 32) T_ = (int)std::min<int64_t>((want + 31) / 32 * 32, 1024);
        RPB_ = T_ >= 32 ? 1 : 256 / T_;
        if (T_ > 32) RPB_ = 1;
        else RPB_ = std::max(1, 256 / T_);
        if (mixed_) {
            // Column sums live in registers beside the row: eight elements of a row per thread where a block can be that wide. Residual +
            // layer norm forward and backward of 8192 x 1024 bfloat16 in one such kernel: 24 us + 4 us for its totals, against 125 us for
            // the nine kernels of one kind of reduction each; bound by instructions in flight and the barriers of four row sums.
            int64_t chunks = std::max<int64_t>(1, 16 / VEC_ / 2);
            auto threads_for = [&](int64_t per_thread) {
                const int64_t t = std::min<int64_t>((nvec + per_thread - 1) / per_thread, 1024);
                int64_t p = 1;
                while (p < t && p < 32) p *= 2;
                return t > 32 ? (t + 31) / 32 * 32 : p;
            };
            const int64_t one = threads_for(1), two = threads_for(2), in_ones = 1024 / one * one, in_twos = 1024 / two * two;
            const bool ones = one == 32 || (one >= 128 && (in_ones > in_twos || in_ones == 1024));
            int64_t warps = 0;  // an SM, at least; otherwise up to 16, 128 registers a thread or more, down to 64 at 1024 threads
            T_ = (int)threads_for(chunks);
            if (min_size == 2 && VEC_ >= 4 && C_ >= 1024 && (C_ <= 2048 || C_ > 3072 || R_ * C_ >= 1 << 21)) {
                // Rows of 16 bits from 1024 columns on: two vectors of eight bytes a thread and as many blocks as 16 warps and more need, so
                // that a block of 13 to 15 warps is not alone on its SM, 24 where every thread has both vectors whole and few sums to keep (84
                // registers do: a layer norm's gradients 16384 x 1024 39.0 -> 32.0, 21845 x 1536 68 -> 61, 16384 x 2048 71 -> 60, the same at
                // 2^22 elements 1.05 - 1.12, with four row sums 1.2, 512 threads 1.06, a last vector that some lack 1.03 - 1.1; operands of
                // float32, which hold twice as much, 0.86 - 0.98 with 128 threads a row, but beyond them 30.9 -> 34.8 at 10922 x 1536). us, the sums
                // above, one vector of 16 bytes a thread -> so: 2048 x 1024 12.9 -> 11.0, 4096 x 2048 32.6 -> 31.8, 3640 x 2304 42 -> 35,
                // 2532 x 3312 52 -> 45, 1677 x 5000 48 -> 41, 1024 x 8192 58 -> 45.
                // Few rows of 2049 to 3072 columns, whose blocks would have nine to twelve warps, are left: 455 x 2304 9.9 against 10.5.
                VEC_ = 4, nvec = vectors(), chunks = 2;
                T_ = (int)threads_for(chunks);
                if (T_ > 288 && T_ <= 384 && C_ % (T_ * 8) != 0) T_ = (int)threads_for(3);  // (the last chunk a part: 2600 wide as fast, few rows faster)
                else warps = !sixteen_warps_ && few_sums() && (!wide_operands() || held_columns() + 2 * wide_operands() <= (T_ <= 128 ? 9 : 8)) && T_ <= 256 && C_ == T_ * VEC_ * 2 && R_ * C_ >= 1 << 23 ? 24 : 16;
            } else if (min_size == 2 && VEC_ == 8 && C_ > 256 && C_ < 1024 && R_ * C_ >= 1 << 20 && !sixteen_warps_) {
                // Rows of 264 to 1016 columns of 16 bits. Up to 384 columns a warp to a row, so that row sums need no barrier between warps, with three
                // vectors of eight bytes a thread and 20 warps an SM; from there two of them a thread and 24 warps, but from 2^21 elements on, where
                // threads hold little, a warp to a row with two or three vectors of 16 bytes: up to 512 columns; beyond them with few row sums where
                // no lane lacks its last vector, and else up to five million elements. Times a vector of 16 bytes a thread and 16 warps, gradients of
                // a layer norm, layer and RMS norm and softmax with theirs, softmax with column sums, 2^20 to 2^25 elements: 0.39 - 1.0. A warp
                // to a row against two vectors a thread, 520, 640, 744 and 760 columns: four million elements 0.90 - 1.07, seven 0.96 - 1.09 (two
                // softmaxes, five row sums, 1.03 - 1.26), nine and more 0.99 - 1.30; 768 columns: one or two row sums 0.89 - 1.02 at any of these
                // sizes, more 0.95 - 1.29.
                chain_ = VEC_;
                const bool warp_rows = C_ <= 512 || (nvec % 32 == 0 ? few_sums() : row_sums() <= 4 && R_ * C_ <= 5 << 20);
                if (C_ > 384 && C_ <= 768 && R_ * C_ > 1 << 21 && warp_rows && held_columns() <= 9) {
                    T_ = 32, warps = C_ <= 512 ? 16 : 12;
                } else {
                    VEC_ = 4, nvec = vectors(), chunks = C_ <= 384 ? 3 : 2;
                    T_ = (int)threads_for(chunks), warps = C_ <= 384 ? 20 : 24;
                }
            } else if (min_size == 4 && VEC_ == 4 && nvec <= 1024 && R_ * C_ >= 1 << 21 && held_columns() <= 16 && (ones || col_reduces_.size() <= 4)) {
                // float32 rows: one vector a thread where that makes a warp or four and more, 32 warps an SM; two where more threads fit so,
                // or as many but not all 1024. us, two vectors and 16 warps -> so: 16384 x 512 44 -> 33, 8192 x 1024 46 -> 35, 5461 x 1536 58 -> 40,
                // 4096 x 2048 50 -> 40, 2532 x 3312 73 -> 55, 2048 x 4096 61 -> 44; fewer than two million elements are up to 1.16 slower.
                // Such threads have 64 registers. 1 to 4 operands with 2 to 12 column sums and none or two operands by column, 2^23 elements, times
                // two vectors and 16 warps: 0.51 - 1.03 within the bound above, 0.95 - 1.23 beyond it; two vectors in 64 to 72 registers (1536 and
                // 3312 columns) 0.74 - 0.96 with up to four column sums, 0.82 - 1.12 with five, 0.82 - 1.29 with eight, 1.1 - 1.8 with more.
                T_ = (int)(ones ? one : two);
                if (T_ >= 128 || one == 32) warps = 32;
            } else if (T_ > 256 && T_ <= 384) {
                // A block of 288 to 384 threads would be alone on its SM with 9 to 12 warps: twelve elements a thread instead make two of
                // 192 to 256. The same sums of 14563 rows: 3001 wide float32 387 -> 244 us, bfloat16 257 -> 214.
                if (VEC_ == 8) VEC_ = 4, nvec = vectors(), chunks = 2;
                T_ = (int)threads_for(chunks * 3 / 2);
            }
            RPB_ = T_ > 32 ? 1 : 128 / T_;
            const int64_t threads = T_ * RPB_;
            resident_ = (int)std::max<int64_t>(1, warps ? std::min((warps * 32 + threads - 1) / threads, 1024 / threads) : 512 / threads);
        }
        if (!mixed_ && !shifted_ && !multi_ && has_reduce_ && VEC_ * min_size == 16) row_residency(nvec);
        NCH_ = (int)((nvec + T_ - 1) / T_);
        if (shifted_) {
            period_ = VEC_;  // (the width is odd)
            // As many blocks as are resident at once, so that each moves the columns' operands into place once for all its rows: 24 warps an
            // SM where rows are summed, else 32. (5590 x 3001, us: 12.0; with as many blocks as an SM has threads for, 2048, 16.4.)
            resident_ = (int)std::max<int64_t>(1, (has_reduce_ ? 768 : 1024) / (T_ * RPB_));
        }
        if (NCH_ > 64) fail(LB_ERR_UNSUPPORTED, format("rows of %lld elements are too long for the fused row kernel", (long long)C_));
        wide_index_ = R_ * C_ >= (1LL << 31) - 4096;
        for (int v : g_.inputs)
            if (g_.type(v).numel() >= (1LL << 31) - 4096) wide_index_ = true;
        if (multi_) wide_index_ = true;  // a group's row count is a run-time value
        pair_ = VEC_ >= 2 && computes_bf16();
    }

    // Threads of a row and blocks an SM of kernels that go over a row more than once, where the compiler's own choice of registers leaves an SM
    // with one block of 256 threads, or rows of many vectors are summed over more threads than those sums are worth (each warp of a row takes
    // part in every total: ten shuffles of 1024 threads' second stage). What decides is what a thread holds of a row: a rule that looked at the
    // width alone made cross entropy of two operands up to 3.1 times as slow, norms of float32 rows beside 16-bit operands up to 2.6. us, as it
    // was -> so, 2^24 elements, bfloat16 where nothing else is said:
    //   norms - rows written by what their sums say and by operands of the columns, no exponential on the way - are built for 512 threads an SM,
    //   768 where a thread has 16 elements. One operand over the space: layer norm of 512 columns 11.3 -> 9.5, 1024 11.4 -> 9.6, 1536 11.8 -> 10.3, 4096
    //   12.7 -> 11.0, float32 21.5 -> 20.3, 22.2 -> 20.7, float32 of three vectors a thread left; rms norm (one sum) up to 1024 columns 10.0 -> 8.6, at
    //   2048 9.2 -> 8.6, but three vectors a thread 8.9 -> 9.6. Several operands: residual + layer norm of 1024 columns 34.8 -> 31.2, 8192 49.5 ->
    //   35.6; left at 64 threads a row and with three vectors a thread (0.92 - 1.11; float32 beside 16 bits with three gains 0.90 - 0.97), at
    //   float32 whose operands and results are four (42.0 -> 45.4: bandwidth), and rows of 16 bits with four vectors a thread, weights of float32 and
    //   32 threads a row (19.8 -> 21.7);
    //   ... of which 512 threads and more walked 16-bit rows: eleven vectors a thread, 1024 threads an SM. Layer norm of 9872 columns 19.9 -> 14.0,
    //   32768 28.5 -> 15.5, rms norm 14.6 -> 9.4, 15.8 -> 10.4. Two operands of 16 bits fit from where threads had four vectors and more: residual +
    //   rms norm of 33000 columns 37.9 -> 27.6, 16384 28.0 -> 26.9 and 9872 24.2 -> 27.8 left; + layer norm 50304 47.8 -> 41.4, 36000 42.2 -> 47.3;
    //   rows that are summed several times and not written (cross entropy), one operand of 16 bits: eleven vectors too, up to 512 threads. 9872
    //   columns 11.8 -> 7.4, 32768 11.2 -> 8.7, but 50304 (608 threads) 9.9 -> 10.6; two operands of 32768 columns 19.1 -> 59.2;
    //   float32 rows of several sums, one operand and none of columns, of which a power of two of threads leaves some idle: four vectors a
    //   thread, two blocks an SM. 8200 columns, softmax 31.2 -> 25.5, cross entropy 24.4 -> 15.2; two operands 25.2 -> 31.0.
    // Others are left: softmax, whose exponentials are taken again for its result, 0.8 - 1.3 of the time on any other threads, log softmax and
    // centred rows 1.0 - 1.4.
    int per_sm_ = 0;
    // Whether an operand is read otherwise than by a gather (cross entropy's logits are, once more)
    bool read_in_rows(int v) const {
        for (const Node& n : g_.nodes)
            for (size_t k = 0; k < n.inputs.size(); k++)
                if (n.inputs[k] == v && !(n.op == "gather" && k == 0)) return true;
        return false;
    }
    void row_residency(int64_t nvec) {
        int sums = 0, behind = 0;
        std::map<int, int> seen;  // of a value: 1 behind a row's sum, 2 from an exponential of the space
        for (const Node& n : g_.nodes) {
            const bool reduce = n.op == "reduce_sum" || n.op == "reduce_max";
            sums += reduce;
            int has = reduce ? 1 : n.op == "exp" ? 2 : 0;
            for (int v : n.inputs)
                if (auto it = seen.find(v); it != seen.end()) has |= reduce ? it->second & 1 : it->second;
            seen[n.output] = has;
        }
        bool written = false, columns = false, wide_columns = false;
        int row_bytes = 0, bytes = 0;  // of an element: of the operands that span the space, of results too
        for (int v : g_.outputs)
            if (g_.type(v).numel() == R_ * C_) written = true, behind |= seen[v], bytes += dtype_size(g_.type(v).dtype);
        for (int v : g_.inputs) {
            const int64_t n = g_.type(v).numel();
            const int size = dtype_size(g_.type(v).dtype);
            if (n == R_ * C_ && read_in_rows(v)) row_bytes += size, bytes += size;
            else if (n == C_ && R_ > 1) columns = true, wide_columns |= size * VEC_ > 16;
        }
        const bool norm = written && behind == 1 && columns, summed = !written && sums > 1, one = row_bytes * VEC_ == 16;
        const int64_t eleven = (nvec * 3 / 32 + 31) / 32 * 32, four = (nvec + 127) / 128 * 32, elements = (nvec + T_ - 1) / T_ * VEC_;
        const int former = T_;
        const bool two = norm && !wide_operands() && row_bytes == 4 && nvec >= (sums == 1 ? 4096 : 5120);
        if (T_ >= 512 && !one && !two) {
        } else if (T_ >= 512 && narrow_) {
            if (norm && eleven <= 1024) T_ = (int)eleven, per_sm_ = std::max(1, 1024 / T_);
            else if (summed && eleven <= 512) T_ = (int)eleven, per_sm_ = (T_ > 256 ? 1536 : 1024) / T_;
        } else if (T_ >= 512) {
            if (sums > 1 && !columns && 8 * four <= 7 * (int64_t)T_) T_ = (int)four, per_sm_ = T_ <= 640 ? 2 : 0;
        } else if (T_ <= 256 && norm && elements >= 16) {
            const bool pays = sums == 1  ? one && (T_ <= 32 || (narrow_ && elements > 24))
                              : !narrow_ ? bytes < 16
                              : one      ? T_ > 32 || elements <= 24 || !wide_columns
                                         : T_ <= 32 || (elements > 24 ? T_ > 64 : row_bytes > 4);
            if (pays) per_sm_ = std::max(1, (elements > 16 ? 512 : 768) / (T_ * RPB_));
        }
        if (T_ < former) chain_ = (int)std::max<int64_t>(VEC_, nvec * VEC_ / former);
    }

    int row_sums() const {
        int sums = -(int)col_reduces_.size();
        for (const Node& n : g_.nodes) sums += n.op == "reduce_sum" || n.op == "reduce_max";
        return sums;
    }
    // Whether a mixed kernel keeps little for a column and for a row
    bool few_sums() const { return row_sums() <= 2 && held_columns() <= 9; }

    // Operands over the space of more than 16 bits
    int wide_operands() const {
        int wide = 0;
        for (int v : g_.inputs) wide += g_.type(v).numel() == R_ * C_ && dtype_size(g_.type(v).dtype) > 2;
        return wide;
    }

    // What a thread of a mixed kernel holds for each of its columns: a sum for each column total, the operands by column, and those over the
    // space twice (the row in flight and the one behind it)
    int held_columns() const {
        int held = (int)col_reduces_.size();
        for (int v : g_.inputs) held += g_.type(v).numel() == R_ * C_ ? 2 : g_.type(v).numel() == C_;
        return held;
    }

    // Whether rows of an odd width are read in whole vectors all the same. Their elements start at any address, but all tensors over
    // the space start alike: a row's chunks begin at the aligned address at or before its first element, and its neighbours' elements
    // in the first and the last chunk count for nothing and are not written. A block walks rows that start at the same distance from an
    // aligned address (every eighth one does), so that a thread keeps its columns. The tensors are read as the space is laid out, by
    // column, by row or as one value; the columns' operands are moved into place once a block.
    // For bfloat16 pairs, one row sum at most and six million elements and more. What bounded such rows was one load and one store an
    // element. Multiply-add-relu with and without a row sum of squares, and a row sum alone, us, 55 shapes of 6.3 to 34 million
    // elements and 129 to 16383 columns, element by element -> so: 0.45 - 1.03 of the time (5590 x 3001 19.2 -> 12.0, 22.0 -> 13.4, 9.2 ->
    // 6.5; 32704 x 513 19.7 -> 18.0; floor at the copy's bandwidth 10.3, 10.3, 5.1). Left as they were: 4 million elements (0.8 - 1.12),
    // several row sums (softmax 1.1 - 1.5: three phases with their masks), float32 (0.8 - 1.3: four bytes a thread are half a line's
    // worth already), float16 (0.9 - 1.6: no pairs), even widths (0.9 - 1.8), column sums in the same kernel (1.0 - 2.0).
    bool shiftable(const TensorType& space, int widest) const {
        if (multi_ || R_ < widest || C_ < kShiftedColumns || R_ * C_ < kShiftedElements) return false;
        int row_sums = 0;
        for (const Node& n : g_.nodes) {
            if (n.op == "gather" || n.op == "iota" || n.op == "slice" || n.op == "transpose") return false;
            row_sums += n.op == "reduce_sum" || n.op == "reduce_max";
        }
        if (row_sums > 1 || !computes_bf16()) return false;
        for (int v : g_.inputs) {
            const TensorType& t = g_.type(v);
            const int64_t n = t.numel();
            const bool spans = n == R_ * C_ && t.shape.back() == space.shape.back(), columns = n == C_ && t.shape.back() == C_;
            if (!spans && !columns && n != R_ && n != 1) return false;
            if (spans && space.shape.back() != C_ && t.shape != space.shape) return false;
        }
        for (int v : g_.outputs) {
            const TensorType& t = g_.type(v);
            if (t.numel() == R_ * C_ && t.shape.back() != space.shape.back()) return false;
        }
        return true;
    }
    static constexpr int64_t kShiftedColumns = 128, kShiftedElements = 6 << 20;
    std::string column() const { return shifted_ ? "column(c0 + e)" : "(c0 + e)"; }

    // Vectors of a row per thread: four of 16 bytes. Of the narrow ones that a width without a power of two allows, 16 (eight of
    // two elements) where rows are long and many: a row over 1024 threads of three 2-byte loads each is bound by its barriers and by
    // loads in flight, and a power of two of threads may leave a quarter to a half of them idle. The multiply-add-relu-square-sum
    // chain, us, 4 -> 16 vectors of one element: 5000 x 3001 bfloat16 21.0 -> 16.6, 20000 x 513 18.5 -> 12.0, 5000 x 1025 10.7 -> 6.7,
    // 100000 x 257 float32 42 -> 36; but 64 x 513 1.8 -> 1.9, 20000 x 511 12.1 -> 14.9, 20000 x 127 4.4 -> 7.0, 100000 x 31 5.4 -> 13.3 and 3 x 255 1.6 -> 3.2.
    // Eight instead of 16 where those are slower: 5000 x 129 4.0 -> 2.8, 100000 x 65 12.7 -> 9.7. Each further reduction of a row (softmax,
    // norms) adds barriers: 5000 x 3001 bfloat16 28.4 -> 14.8, 20000 x 511 12.8 -> 8.5. Rows without a reduction: 20000 x 1025 18.7 -> 16.2,
    // 64 x 2047 1.4 -> 1.7.
    int64_t vectors_per_thread(int64_t nvec) const {
        if (VEC_ > 2) return 4;
        if (!has_reduce_) return R_ * nvec >= 1 << 19 ? 16 / VEC_ : 4;
        int row_sums = 0;
        for (const Node& n : g_.nodes) row_sums += n.op == "reduce_sum" || n.op == "reduce_max";
        const bool several = row_sums > 1;
        if (R_ < (nvec > 1024 ? 256 : 512)) return 4;
        if (VEC_ == 2) return nvec > (several ? 256 : 512) ? 8 : 4;
        int64_t threads = 1;
        while (threads < (nvec + 3) / 4) threads *= 2;
        const bool idle = nvec * 4 < 3 * threads * ((nvec + threads - 1) / threads);  // over a quarter, with four vectors a thread
        if (nvec > 1024 || (nvec > 256 && (idle || (several && R_ >= 4096))) || (nvec > 768 && (several || R_ >= 4096)) || (nvec > 96 && idle && several && R_ >= 4096)) return 16;
        if ((nvec > 128 && nvec <= 256) || (nvec > 64 && idle && R_ >= (several ? 4096 : 16384))) return 8;
        return 4;
    }

    // pair mode pays where packed bfloat16 instructions replace scalar ones
    bool computes_bf16() const {
        for (const Node& n : g_.nodes)
            if (g_.type(n.output).dtype == LB_BF16) return true;
        for (int v : g_.inputs)
            if (g_.type(v).dtype == LB_BF16) return true;
        return false;
    }

    Comp row_comp() {
        Comp c;
        c.expr = "r";
        c.row_dep = true;
        return c;
    }
    Comp col_comp() {
        Comp c;
        c.expr = column();
        c.base = "c0";
        c.lane = !shifted_;
        c.e_dep = c.c_dep = true;
        return c;
    }

    // Drops redundant outer parentheses, "((r))" -> "r", so that the same coordinate reached through different
    // reshapes gets the same text: values and reductions are memoised by the text of their index.
    static std::string tidy(std::string s) {
        for (;;) {
            if (s.size() < 2 || s.front() != '(' || s.back() != ')') return s;
            int depth = 0;
            bool wraps = true;
            for (size_t k = 0; k + 1 < s.size(); k++) {
                if (s[k] == '(') depth++;
                if (s[k] == ')' && --depth == 0) wraps = false;
            }
            if (!wraps) return s;
            std::string inner = s.substr(1, s.size() - 2);
            bool simple = !inner.empty();
            for (char c : inner) simple &= ident_char(c);
            bool wrapped_again = inner.size() >= 2 && inner.front() == '(' && inner.back() == ')';
            if (wrapped_again) {
                int d = 0;
                for (size_t k = 0; k + 1 < inner.size(); k++) {
                    if (inner[k] == '(') d++;
                    if (inner[k] == ')' && --d == 0) wrapped_again = false;
                }
            }
            if (!simple && !wrapped_again) return s;
            s = inner;
        }
    }

    // coordinates of flat index `flat` in `shape`
    Index unravel(const Comp& flat, const std::vector<int64_t>& shape) {
        Index out(shape.size());
        int rank = (int)shape.size();
        bool keep_lane = flat.lane && rank > 0 && shape[rank - 1] % VEC_ == 0;
        int64_t stride = 1;
        for (int d = rank - 1; d >= 0; d--) {
            Comp c;
            c.row_dep = flat.row_dep;
            c.dyn = flat.dyn;
            c.c_dep = flat.c_dep;
            if (shape[d] == 1) {
                c = zero_comp();
            } else {
                const std::string src = tidy(keep_lane ? flat.base : flat.expr);
                std::string q = stride == 1 ? src : format("(%s / %lld)", src.c_str(), (long long)stride);
                // the leading coordinate needs no modulo: the flat index is in range
                std::string coord = d == 0 ? q : format("(%s %% %lld)", q.c_str(), (long long)shape[d]);
                if (keep_lane && d == rank - 1) {
                    c.base = coord;
                    c.expr = format("(%s + e)", coord.c_str());
                    c.lane = c.e_dep = true;
                } else {
                    c.expr = coord;
                    c.e_dep = keep_lane ? false : flat.e_dep;
                }
            }
            out[d] = c;
            stride *= shape[d];
        }
        return out;
    }

    Comp ravel(const Index& idx, const std::vector<int64_t>& shape) {
        Comp out;
        int rank = (int)shape.size();
        if (rank == 0) return zero_comp();
        bool lane = idx[rank - 1].lane && (rank == 1 || shape[rank - 1] % VEC_ == 0);
        for (int d = 0; d < rank - 1; d++)
            if (idx[d].e_dep) lane = false;
        std::string sum;
        int64_t stride = numel(shape);
        for (int d = 0; d < rank; d++) {
            stride /= std::max<int64_t>(shape[d], 1);
            const Comp& c = idx[d];
            out.row_dep |= c.row_dep;
            out.dyn |= c.dyn;
            out.c_dep |= c.c_dep;
            out.e_dep |= c.e_dep;
            if (c.zero_known || shape[d] == 1) continue;
            std::string term = (lane && d == rank - 1) ? c.base : c.expr;
            if (stride != 1) term = format("(idx_t)%s * %lld", term.c_str(), (long long)stride);
            sum += (sum.empty() ? "" : " + ") + term;
        }
        if (sum.empty()) sum = "0";
        if (lane) {
            out.lane = true;
            out.base = tidy("(" + sum + ")");
            out.expr = "(" + sum + " + e)";
        } else {
            out.expr = tidy("(" + sum + ")");
        }
        if (out.expr == "0") return zero_comp();
        return out;
    }

    Index output_index(const TensorType& t, bool full) {
        if (!full) return unravel(row_comp(), t.shape);
        if (t.rank() >= 1 && t.shape.back() == C_) {
            std::vector<int64_t> lead(t.shape.begin(), t.shape.end() - 1);
            Index idx = unravel(row_comp(), lead);
            idx.push_back(col_comp());
            return idx;
        }
        Comp flat;
        flat.base = format("(r * (idx_t)%lld + c0)", (long long)C_);
        flat.expr = shifted_ ? format("(r * (idx_t)%lld + %s)", (long long)C_, column().c_str()) : format("(r * (idx_t)%lld + c0 + e)", (long long)C_);
        flat.lane = !shifted_;
        flat.e_dep = flat.c_dep = flat.row_dep = true;
        return unravel(flat, t.shape);
    }

    static std::string key_of(int v, const Index& idx) {
        std::string k = std::to_string(v);
        for (const Comp& c : idx) k += "|" + c.expr;
        return k;
    }
    static bool e_dep(const Index& idx) {
        for (const Comp& c : idx)
            if (c.e_dep) return true;
        return false;
    }
    static bool c_dep(const Index& idx) {
        for (const Comp& c : idx)
            if (c.c_dep) return true;
        return false;
    }

    // ---- pair mode -----------------------------------------------------------------------------------------
    // The element loop advances two elements per step. A value that depends on the element is a pair variable
    // (p2<T>, or packed bf16x2); its defining expression is written once with operand placeholders @k@ and
    // instantiated for lane 0 and lane 1. Values that do not depend on the element stay scalars.
    bool pair_ = false;
    std::map<std::string, int> pair_vars_;  // pair variable -> dtype (-1 for index variables)
    std::set<std::string> body_names_;      // otherwise: the variables of the loops over elements

    static bool ident_char(char c) { return std::isalnum((unsigned char)c) || c == '_'; }
    static bool mentions_e(const std::string& s) {
        for (size_t k = 0; k < s.size(); k++)
            if (s[k] == 'e' && (k == 0 || !ident_char(s[k - 1])) && (k + 1 == s.size() || !ident_char(s[k + 1]))) return true;
        return false;
    }
    // `expr` for lane 0 or 1: placeholders become L<lane>(operand), LX( becomes L<lane>(, the element index e
    // becomes (e + 1) in lane 1
    static std::string lane_of(const std::string& expr, int lane, const std::vector<std::string>* ops) {
        std::string a;
        const char* acc = lane ? "L1(" : "L0(";
        for (size_t k = 0; k < expr.size(); k++) {
            if (expr[k] == '@') {
                size_t end = expr.find('@', k + 1);
                int which = std::stoi(expr.substr(k + 1, end - k - 1));
                a += acc + (*ops)[which] + ")";
                k = end;
            } else if (expr.compare(k, 3, "LX(") == 0 && (k == 0 || !ident_char(expr[k - 1]))) {
                a += acc;
                k += 2;
            } else {
                a += expr[k];
            }
        }
        if (!lane) return a;
        std::string out;
        for (size_t k = 0; k < a.size(); k++) {
            if (a[k] == 'e' && (k == 0 || !ident_char(a[k - 1])) && (k + 1 == a.size() || !ident_char(a[k + 1]))) out += "(e + 1)";
            else out += a[k];
        }
        return out;
    }
    // a statement per lane (accumulations, stores)
    static std::string both_lanes(const std::string& stmt) { return lane_of(stmt, 0, nullptr) + lane_of(stmt, 1, nullptr); }
    static std::string whole_of(const std::string& expr, const std::vector<std::string>* ops) {
        std::string a;
        for (size_t k = 0; k < expr.size(); k++) {
            if (expr[k] == '@') {
                size_t end = expr.find('@', k + 1);
                a += (*ops)[std::stoi(expr.substr(k + 1, end - k - 1))];
                k = end;
            } else {
                a += expr[k];
            }
        }
        return a;
    }
    // an operand usable by a packed bf16x2 instruction: a packed pair, or a scalar that is the same for both lanes
    bool packable(const std::string& operand, int dtype = LB_BF16) const {
        auto it = pair_vars_.find(operand);
        if (it != pair_vars_.end()) return it->second == dtype;
        return !mentions_e(operand) && operand.find("LX(") == std::string::npos;
    }
    bool pairs_here(const Phase& ph, bool in_body) const { return pair_ && in_body && ph.chunked; }

    // Defines a variable holding `expr` in the right scope of `ph` and returns its name. In pair mode `ops` are the
    // operands behind the placeholders; `whole` marks an expression that already yields a packed bf16x2.
    std::string define(Phase& ph, const char* type, const std::string& expr, bool in_body,
                       const std::vector<std::string>* ops = nullptr, int dtype = -1, bool whole = false) {
        std::string name = fresh("v");
        if (!pairs_here(ph, in_body)) {
            std::string line = format("%s %s = %s;\n", type, name.c_str(), expr.c_str());
            (in_body && ph.chunked ? ph.body : ph.pre) += line;
            if (in_body && ph.chunked) ph.body_vars.push_back({type, name, ph.parts.size()}), body_names_.insert(name);
            return name;
        }
        if (whole) {
            ph.body += format("%s %s = %s;\n", dtype == LB_BF16 ? "bf16x2" : "p2<float>", name.c_str(), whole_of(expr, ops).c_str());
        } else if (dtype == LB_BF16) {
            // one packed conversion rounds both lanes; values that already are bf16 are packed by their bits
            static const std::string rnd = "rnd_bf16(";
            bool rounds = expr.compare(0, rnd.size(), rnd) == 0 && expr.back() == ')';
            if (rounds) {
                int depth = 0;
                for (size_t k = rnd.size() - 1; k < expr.size(); k++) {
                    if (expr[k] == '(') depth++;
                    if (expr[k] == ')' && --depth == 0 && k + 1 != expr.size()) rounds = false;
                }
            }
            std::string inner = rounds ? expr.substr(rnd.size(), expr.size() - rnd.size() - 1) : expr;
            ph.body += format("bf16x2 %s = %s(%s, %s);\n", name.c_str(), rounds ? "mk_bf16x2" : "pk_bf16x2",
                              lane_of(inner, 0, ops).c_str(), lane_of(inner, 1, ops).c_str());
        } else {
            ph.body += format("p2<%s> %s = {%s, %s};\n", type, name.c_str(), lane_of(expr, 0, ops).c_str(), lane_of(expr, 1, ops).c_str());
        }
        pair_vars_[name] = dtype;
        ph.body_vars.push_back({dtype == LB_BF16 ? "bf16x2" : whole ? std::string("p2<float>") : format("p2<%s>", type), name, ph.parts.size()});
        return name;
    }

    // Whether values are exponentials, or products and quotients of one: next to nothing for some elements (a softmax's terms, its
    // probabilities), so that they would be divided as usual after all. us, divided by the row's sum as chunks -> one by one: float32
    // softmax of 32768 x 1024 standard normal logits 43.1 -> 43.4, logits that spread by 80 64 -> 51, by 170 209 -> 196.
    std::map<int, bool> tiny_;
    bool may_be_tiny(int v) {
        const Node* n = g_.node_of(v);
        if (!n) return false;
        if (auto it = tiny_.find(v); it != tiny_.end()) return it->second;
        static const std::set<std::string> carry = {"mul", "select", "neg", "abs", "cast", "reshape", "broadcast_in_dim"};
        bool tiny = n->op == "exp";
        if (n->op == "div") tiny = may_be_tiny(n->inputs[0]);
        else if (carry.count(n->op)) tiny = std::any_of(n->inputs.begin(), n->inputs.end(), [&](int in) { return may_be_tiny(in); });
        return tiny_[v] = tiny;
    }

    // Whether a division of float32 elements by `divisor` is one by the same value for the whole chunk. (Blocks of 800 threads and more
    // with float32 rows and their column sums have no registers left for it: 7360 wide 1.05 to 1.1 of the time.)
    bool divides_chunk(const Phase& ph, const std::string& dividend, const std::string& divisor, bool pairs) const {
        if (column_mode_ || multi_ || VEC_ < 4 || (mixed_ && T_ > 768 && NCH_ > 1 && !narrow_) || !ph.chunked || mentions_e(divisor) || divisor.find("LX(") != std::string::npos) return false;
        if (!pairs) return body_names_.count(dividend) && !body_names_.count(divisor);
        auto it = pair_vars_.find(dividend);
        return it != pair_vars_.end() && it->second == LB_F32 && !pair_vars_.count(divisor);
    }
    // `dividend / divisor` as one division of the whole chunk, and the variable that holds the quotient in the loop over its elements.
    std::string chunk_quotient(Phase& ph, const std::string& key, const std::string& dividend, const std::string& divisor, bool pairs) {
        const char* type = pairs ? "p2<float>" : "float";
        const char* at = pairs ? "e / 2" : "e";
        const std::string num = fresh("num"), quo = fresh("quo"), count = pairs ? "VEC / 2" : "VEC";
        std::string& y = ph.memo["rcp|" + divisor];
        if (y.empty()) {
            y = fresh("rcp");
            ph.pre += format("const float %s = row_reciprocal(%s);\n", y.c_str(), divisor.c_str());
        }
        ph.chunk_decls += format("%s %s[%s];\n", type, num.c_str(), count.c_str());
        ph.body += format("%s[%s] = %s;\n", num.c_str(), at, dividend.c_str());
        auto known = quotients_.find(dividend);  // of the same divisor: no other quotient's range is known here
        const bool again = known != quotients_.end() && known->second.second == y;
        const std::string range = again ? ", " + known->second.first + "_range" : "";
        ph.parts.push_back({ph.body, format("%s_range = %s<%s>(%s, %s, %s, %s%s);\n", quo.c_str(), again ? "divide_again" : "divide_chunk", count.c_str(), num.c_str(), quo.c_str(), divisor.c_str(), y.c_str(), range.c_str()), key, quo, type});
        ph.body.clear();
        const std::string name = fresh("v");
        ph.body += format("const %s %s = %s[%s];\n", type, name.c_str(), quo.c_str(), at);
        ph.body_vars.push_back({type, name, ph.parts.size()});
        quotients_[name] = {quo, y};
        if (pairs) pair_vars_[name] = LB_F32;
        else body_names_.insert(name);
        return name;
    }
    std::map<std::string, std::pair<std::string, std::string>> quotients_;  // a chunk quotient's variable -> its array, the reciprocal
    static bool mentions(const std::string& code, const std::string& name) {
        for (size_t at = code.find(name); at != std::string::npos; at = code.find(name, at + 1))
            if ((at == 0 || !ident_char(code[at - 1])) && (at + name.size() == code.size() || !ident_char(code[at + name.size()]))) return true;
        return false;
    }
    // The loops over a chunk's elements: one, or one per part with variables that later parts read handed on in arrays. Called for the
    // phases in the order in which they run: rows of few elements a thread keep their quotients for the phases that divide the same again.
    std::map<std::string, std::string> kept_quotients_;  // value and index -> array
    std::string element_loops(const Phase& ph) {
        std::vector<Phase::Part> parts = ph.parts;
        const std::string at = pair_ ? "e / 2" : "e";
        std::string decls = ph.chunk_decls;
        for (Phase::Part& part : parts) {
            const std::string count = pair_ ? "VEC / 2" : "VEC";
            if (!has_reduce_ || NCH_ * VEC_ > 16) {
                decls += format("%s %s[%s];\nMagnitudes %s_range;\n", part.type.c_str(), part.array.c_str(), count.c_str(), part.array.c_str());
                continue;
            }
            auto [kept, first] = kept_quotients_.emplace(part.key, part.array + "_row");
            if (first) row_decls_ += format("%s %s[NCH][%s];\nMagnitudes %s_range[NCH];\n", part.type.c_str(), kept->second.c_str(), count.c_str(), kept->second.c_str());
            else part.then.clear();
            decls += format("auto& %s = %s[ch];\nauto& %s_range = %s_range[ch];\n", part.array.c_str(), kept->second.c_str(), part.array.c_str(), kept->second.c_str());
        }
        parts.push_back({ph.body, "", "", "", ""});
        for (const Phase::BodyVar& v : ph.body_vars) {
            bool later = false;
            for (size_t k = v.part + 1; k < parts.size(); k++)
                if (mentions(parts[k].body, v.name)) {
                    parts[k].body = format("const %s %s = %s_all[%s];\n", v.type.c_str(), v.name.c_str(), v.name.c_str(), at.c_str()) + parts[k].body;
                    later = true;
                }
            if (!later) continue;
            decls += format("%s %s_all[%s];\n", v.type.c_str(), v.name.c_str(), pair_ ? "VEC / 2" : "VEC");
            parts[v.part].body += format("%s_all[%s] = %s;\n", v.name.c_str(), at.c_str(), v.name.c_str());
        }
        std::string out = decls;
        for (const Phase::Part& part : parts) {
            if (!part.body.empty())
                out += format("#pragma unroll\nfor (int e = 0; e < VEC; e += %d) {\n", pair_ ? 2 : 1) + indent(part.body, 4) + "}\n";
            out += part.then;
        }
        return out;
    }

    // the statement(s) placing element e (and e + 1 in pair mode) of `val` in the staging array `buf`
    std::string store_element(const std::string& buf, int dtype, const std::string& val) {
        if (!pair_) return format("%s[e] = %s;\n", buf.c_str(), to_memory(dtype, val).c_str());
        auto it = pair_vars_.find(val);
        if (it != pair_vars_.end() && it->second == LB_BF16 && dtype == LB_BF16) return format("*(u32*)&%s[e] = %s.v;\n", buf.c_str(), val.c_str());
        return both_lanes(format("%s[e] = %s;\n", buf.c_str(), to_memory(dtype, "LX(" + val + ")").c_str()));
    }
    // Whether a pair's elements are added by one packed instruction: float32 sums. Half the instructions, and a chain half as long. Not in kernels that
    // sum columns and, three times and more, rows: 31 sizes from 8065 x 520 to 8192 x 2048, packed -> an element each, layer norm with its gradients 0.95 - 1.02
    // of the time (21845 x 768 37.2 -> 35.6 us, 5461 x 1536 20.2 -> 19.6, 8192 x 1024 the same), softmax with its gradient 0.97 - 1.01 (16384 x 1024 32.4 -> 31.7),
    // but RMS norm, which sums a row twice, 0.99 - 1.03.
    bool adds_pairs(const std::string& combine, const std::string& val) const {
        return pair_ && !shifted_ && !(mixed_ && row_sums() > 2) && combine == "rnd_f32(__fadd_rn(%A, %B))" && packable(val, LB_F32);
    }
    // the statement(s) folding element e (and e + 1) of `val` into `acc`
    std::string accumulate(const std::string& acc, const std::string& combine, const std::string& val) {
        const char* counts = shifted_ ? "if (whole || in_row(c0 + e)) " : "";  // (a row's neighbours do not)
        if (adds_pairs(combine, val)) {
            const std::string second = lane_of(acc, 1, nullptr);
            return format("{ const p2<float> sum = f32x2_add(p2<float>{%s, %s}, to_f32x2(%s)); %s = sum.x, %s = sum.y; }\n", acc.c_str(), second.c_str(),
                          val.c_str(), acc.c_str(), second.c_str());
        }
        if (!pair_) return format("%s%s = %s;\n", counts, acc.c_str(), subst(combine, acc, val).c_str());
        return both_lanes(format("%s%s = %s;\n", counts, acc.c_str(), subst(combine, acc, "LX(" + val + ")").c_str()));
    }

    // ---- loads ------------------------------------------------------------------------------------------
    std::string vector_element_;  // set by load_input: the staged array element (memory type) when the load is vectorised
    std::string load_input(int position, int v, const Index& idx, Phase& ph) {
        vector_element_.clear();
        const TensorType& t = g_.type(v);
        CType ct = ctype(t.dtype);
        Comp flat = ravel(idx, t.shape);
        std::string ptr = format("((const %s*)in%d)", ct.memory, position);
        const char* plain = inplace_ ? "_plain" : "";
        auto vector_load = [&](const std::string& dst) {
            if (!shifted_) return format("ldv%s<%s, VEC>(%s + %s, %s);", plain, ct.memory, ptr.c_str(), flat.base.c_str(), dst.c_str());
            if (flat.row_dep) return format("ldv_within%s<%s, VEC, idx_t>(%s, %s, (idx_t)%lldLL, %s);", plain, ct.memory, ptr.c_str(), flat.base.c_str(), (long long)(R_ * C_), dst.c_str());
            return format("ldv_shifted<%s, VEC, idx_t>(%s, c0 + shift, shift, (idx_t)NCOLS, %s);", ct.memory, ptr.c_str(), dst.c_str());
        };
        if (shifted_ && ph.chunked && e_dep(idx)) {
            if (t.numel() == R_ * C_ && key_of(0, idx) == key_of(0, output_index(t, true))) {
                flat.lane = true, flat.base = format("(r * (idx_t)%lldLL + c0)", (long long)C_);
            } else if (t.numel() == C_ && flat.expr == "(" + column() + ")" && !inplace_) {
                flat.lane = true, flat.base = "c0";
            }
        }
        if (flat.lane && ph.chunked) {
            // contiguous along the vector lane: one vector load per chunk
            bool column_only = !flat.row_dep && !flat.dyn && !column_mode_;  // same for every row: cache once per CTA
            bool cache_row = !column_only && !flat.dyn && !column_mode_ && multi_phase_hint_ && cached_regs_ + NCH_ * VEC_ <= 96;
            std::string key = format("in%d|%s", position, flat.base.c_str());
            if (column_only && cached_regs_ + NCH_ * VEC_ <= 128) {
                auto it = cached_loads_.find(key);
                if (it == cached_loads_.end()) {
                    std::string buf = fresh("col");
                    kernel_cache_ += format("__align__(16) %s %s[NCH][VEC];\n", ct.memory, buf.c_str());
                    kernel_cache_ += "CHUNK_LOOP_BEGIN " + vector_load(buf + "[ch]") + " CHUNK_LOOP_END\n";
                    cached_regs_ += NCH_ * VEC_ * std::max(1, dtype_size(t.dtype) / 4);
                    it = cached_loads_.emplace(key, buf).first;
                }
                vector_element_ = format("%s[ch][e]", it->second.c_str());
                return from_memory(t.dtype, vector_element_);
            }
            if (cache_row) {
                auto it = cached_loads_.find(key);
                if (it == cached_loads_.end()) {
                    std::string buf = fresh("row");
                    row_cache_ += format("__align__(16) %s %s[NCH][VEC];\n", ct.memory, buf.c_str());
                    row_cache_ += "CHUNK_LOOP_BEGIN " + vector_load(buf + "[ch]") + " CHUNK_LOOP_END\n";
                    row_caches_.push_back({ct.memory, buf, "CHUNK_LOOP_BEGIN " + vector_load(buf + "_nx[ch]") + " CHUNK_LOOP_END\n", NCH_ * VEC_ * dtype_size(t.dtype)});
                    cached_regs_ += NCH_ * VEC_ * std::max(1, dtype_size(t.dtype) / 4);
                    it = cached_loads_.emplace(key, buf).first;
                }
                vector_element_ = format("%s[ch][e]", it->second.c_str());
                return from_memory(t.dtype, vector_element_);
            }
            std::string pkey = "ld|" + key;
            auto it = ph.memo.find(pkey);
            if (it == ph.memo.end()) {
                std::string buf = fresh("ld");
                ph.pre += format("__align__(16) %s %s[VEC]; %s\n", ct.memory, buf.c_str(), vector_load(buf).c_str());
                it = ph.memo.emplace(pkey, buf).first;
            }
            vector_element_ = format("%s[e]", it->second.c_str());
            return from_memory(t.dtype, vector_element_);
        }
        return from_memory(t.dtype, format(inplace_ ? "(*(%s + %s))" : "__ldg(%s + %s)", ptr.c_str(), flat.expr.c_str()));
    }

    bool multi_phase_hint_ = false;
    bool mixed_ = false;         // row and column reductions (or full outputs beside column reductions) in one kernel
    bool column_mode_ = false;   // reductions over the leading axes: partial sums per row slice, then a finalize pass
    bool inplace_ = false;       // an output aliases an input: plain loads, no __restrict__
    bool multi_ = false;         // one launch serves a table of tensor groups: pointers and row count per group
    std::vector<int> col_reduces_;  // values reduced over the leading axes, in node order
    int lead_rank_ = 0;

    // ---- values -----------------------------------------------------------------------------------------
    std::string gen(int v, const Index& idx, Phase& ph) {
        std::string key = key_of(v, idx);
        auto it = ph.memo.find(key);
        if (it != ph.memo.end()) return it->second;
        std::string name = gen_uncached(v, idx, ph);
        ph.memo[key] = name;
        return name;
    }

    // the index of a column reduction's operand at row r, column c0 + e
    Index column_operand_index(const TensorType& x, size_t lead_rank) {
        Comp flat_c;
        flat_c.base = "c0", flat_c.expr = "(c0 + e)";
        flat_c.lane = flat_c.e_dep = flat_c.c_dep = true;
        Index idx = unravel(row_comp(), std::vector<int64_t>(x.shape.begin(), x.shape.begin() + lead_rank));
        Index tail = unravel(flat_c, std::vector<int64_t>(x.shape.begin() + lead_rank, x.shape.end()));
        idx.insert(idx.end(), tail.begin(), tail.end());
        return idx;
    }

    // exp(a - m) with m a row maximum computed in this kernel (through reshapes / broadcasts), read by reduce_sum only
    bool normaliser_term(const Node& n) const {
        if (n.op != "exp" || g_.type(n.output).dtype != LB_F32) return false;
        const Node* sub = g_.node_of(n.inputs[0]);
        if (!sub || sub->op != "sub") return false;
        const Node* m = g_.node_of(sub->inputs[1]);
        while (m && (m->op == "broadcast_in_dim" || m->op == "reshape")) m = g_.node_of(m->inputs[0]);
        if (!m || m->op != "reduce_max") return false;
        // the maximum is taken over the values the difference is formed from (possibly widened first)
        int a = sub->inputs[0], x = m->inputs[0];
        if (a != x) return false;
        bool summed = false;
        for (const Node& u : g_.nodes)
            for (int in : u.inputs)
                if (in == n.output) {
                    if (u.op != "reduce_sum") return false;
                    summed = true;
                }
        for (int out : g_.outputs)
            if (out == n.output) return false;
        return summed;
    }

    std::string gen_uncached(int v, const Index& idx, Phase& ph) {
        const TensorType& t = g_.type(v);
        if ((int)idx.size() != t.rank()) fail(LB_ERR_INVALID, "internal: index rank mismatch");
        CType ct = ctype(t.dtype);
        const Node* n = g_.node_of(v);
        bool in_body = e_dep(idx);
        const bool pairs = pairs_here(ph, in_body);
        if (!n) {
            int position = (int)(std::find(g_.inputs.begin(), g_.inputs.end(), v) - g_.inputs.begin());
            std::string loaded = load_input(position, v, idx, ph);
            if (pairs && t.dtype == LB_BF16 && !vector_element_.empty())
                return define(ph, ct.compute, "ld_bf16x2(&" + vector_element_ + ")", in_body, nullptr, t.dtype, true);
            return define(ph, ct.compute, loaded, in_body, nullptr, t.dtype);
        }
        const std::string& op = n->op;
        // In pair mode operands are referred to by placeholders and instantiated per lane by define().
        std::vector<std::string> ops;
        auto operand = [&](const std::string& name) {
            if (!pairs) return name;
            ops.push_back(name);
            return format("@%d@", (int)ops.size() - 1);
        };
        auto arg = [&](int k) { return operand(gen(n->inputs[k], idx, ph)); };
        auto def = [&](const char* type, const std::string& e, bool body, bool whole = false) {
            return define(ph, type, e, body, &ops, (int)t.dtype, whole);
        };
        const bool packed = pairs && t.dtype == LB_BF16;
        bool flt = dtype_is_float(t.dtype);
        const char* rnd = rnd_fn(t.dtype);
        bool f64 = t.dtype == LB_F64;

        if (op == "add" || op == "sub" || op == "mul" || op == "div" || op == "max" || op == "min" || op == "rem" ||
            op == "pow") {
            std::string a = arg(0), b = arg(1), e;
            if (packed && (op == "add" || op == "sub" || op == "mul" || op == "max" || op == "min") && packable(ops[0]) && packable(ops[1]))
                return def(ct.compute, format("bf16x2_%s(to_bf16x2(%s), to_bf16x2(%s))", op.c_str(), a.c_str(), b.c_str()), in_body, true);
            if (pairs && t.dtype == LB_F32 && (op == "add" || op == "sub" || op == "mul") && packable(ops[0], LB_F32) && packable(ops[1], LB_F32)) {
                if (op != "sub" && ops[1] < ops[0]) std::swap(a, b);  // x * y and y * x are one value
                return def(ct.compute, format("f32x2_%s(to_f32x2(%s), to_f32x2(%s))", op.c_str(), a.c_str(), b.c_str()), in_body, true);
            }
            if (op == "div" && t.dtype == LB_F32 && in_body && !may_be_tiny(n->inputs[0]) && divides_chunk(ph, pairs ? ops[0] : a, pairs ? ops[1] : b, pairs))
                return chunk_quotient(ph, key_of(v, idx), pairs ? ops[0] : a, pairs ? ops[1] : b, pairs);
            if (flt) {
                if (op == "add") e = f64 ? a + " + " + b : "__fadd_rn(" + a + ", " + b + ")";
                else if (op == "sub") e = f64 ? a + " - " + b : "__fsub_rn(" + a + ", " + b + ")";
                else if (op == "mul") e = f64 ? a + " * " + b : "__fmul_rn(" + a + ", " + b + ")";
                else if (op == "div") e = f64 ? a + " / " + b : "__fdiv_rn(" + a + ", " + b + ")";
                else if (op == "max") e = "fmax_nan(" + a + ", " + b + ")";
                else if (op == "min") e = "fmin_nan(" + a + ", " + b + ")";
                else if (op == "rem") e = f64 ? "fmod(" + a + ", " + b + ")" : "fmodf(" + a + ", " + b + ")";
                else e = f64 ? "pow(" + a + ", " + b + ")" : "powf(" + a + ", " + b + ")";
                if (op != "max" && op != "min") e = std::string(rnd) + "(" + e + ")";
            } else {
                std::string T = ct.compute, U = ct.unsigned_t;
                // a constant 0 - x or x * -1 is a negation to the compiler: written RT_ZERO - x like `neg` (see RT_ZERO)
                const std::string zero = "((" + T + ")0LL)", minus_one = "((" + T + ")-1LL)";
                if (op == "add") e = "(" + T + ")((" + U + ")" + a + " + (" + U + ")" + b + ")";
                else if (op == "sub") e = "(" + T + ")((" + U + ")" + (a == zero ? std::string("RT_ZERO") : a) + " - (" + U + ")" + b + ")";
                else if (op == "mul" && (a == minus_one || b == minus_one)) e = "(" + T + ")((" + U + ")RT_ZERO - (" + U + ")" + (a == minus_one ? b : a) + ")";
                else if (op == "mul") e = "(" + T + ")((" + U + ")" + a + " * (" + U + ")" + b + ")";
                else if (op == "div") e = "idiv<" + T + ", " + U + ">(" + a + ", " + b + ")";
                else if (op == "rem") e = "irem<" + T + ">(" + a + ", " + b + ")";
                else if (op == "max") e = "imax<" + T + ">(" + a + ", " + b + ")";
                else if (op == "min") e = "imin<" + T + ">(" + a + ", " + b + ")";
                else fail(LB_ERR_UNSUPPORTED, op + " of integers");
            }
            return def(ct.compute, e, in_body);
        }
        if (op == "and" || op == "or" || op == "xor") {
            const char* sym = op == "and" ? "&" : op == "or" ? "|" : "^";
            std::string e = t.dtype == LB_BOOL ? format("(%s %s %s)", arg(0).c_str(), op == "and" ? "&&" : op == "or" ? "||" : "!=", arg(1).c_str())
                                               : format("(%s)(%s %s %s)", ct.compute, arg(0).c_str(), sym, arg(1).c_str());
            return def(ct.compute, e, in_body);
        }
        if (op == "eq" || op == "lt") {
            return def("bool", format("(%s %s %s)", arg(0).c_str(), op == "eq" ? "==" : "<", arg(1).c_str()), in_body);
        }
        if (op == "neg") {
            std::string a = arg(0);
            if (packed && packable(ops[0])) return def(ct.compute, "bf16x2_neg(to_bf16x2(" + a + "))", in_body, true);
            if (pairs && t.dtype == LB_F32 && packable(ops[0], LB_F32)) return def(ct.compute, "f32x2_mul(to_f32x2(" + a + "), to_f32x2(-1.0f))", in_body, true);
            return def(ct.compute, flt ? "-" + a : format("(%s)((%s)RT_ZERO - (%s)%s)", ct.compute, ct.unsigned_t, ct.unsigned_t, a.c_str()), in_body);
        }
        if (op == "abs" || op == "sign" || op == "not") {
            std::string a = arg(0), e;
            if (packed && op == "abs" && packable(ops[0])) return def(ct.compute, "bf16x2_abs(to_bf16x2(" + a + "))", in_body, true);
            if (op == "abs") e = flt ? (f64 ? "fabs(" + a + ")" : "fabsf(" + a + ")") : format("(%s)(%s < 0 ? (%s)RT_ZERO - (%s)%s : (%s)%s)", ct.compute, a.c_str(), ct.unsigned_t, ct.unsigned_t, a.c_str(), ct.unsigned_t, a.c_str());
            else if (op == "sign") e = flt ? format("((%s == 0 || %s != %s) ? %s : (%s < 0 ? (%s)-1 : (%s)1))", a.c_str(), a.c_str(), a.c_str(), a.c_str(), a.c_str(), ct.compute, ct.compute) : format("(%s)((%s > 0) - (%s < 0))", ct.compute, a.c_str(), a.c_str());
            else e = t.dtype == LB_BOOL ? "!" + a : format("(%s)~%s", ct.compute, a.c_str());
            return def(ct.compute, e, in_body);
        }
        if (op == "exp" || op == "log" || op == "sqrt" || op == "tanh" || op == "logistic" || op == "rsqrt" ||
            op == "floor" || op == "ceil" || op == "exp2" || op == "log2" || op == "sin" || op == "cos") {
            std::string a = arg(0), e;
            if (f64) {
                if (op == "logistic") e = "1.0 / (1.0 + exp(-" + a + "))";
                else if (op == "rsqrt") e = "1.0 / sqrt(" + a + ")";
                else e = op + "(" + a + ")";
            } else {
                if (op == "logistic") e = "__fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-" + a + ")))";
                else if (op == "rsqrt") e = "__fdiv_rn(1.0f, __fsqrt_rn(" + a + "))";
                else if (op == "sqrt") e = "__fsqrt_rn(" + a + ")";
                else if (normaliser_term(*n)) e = "exp_sum_term(" + a + ")";
                else e = op + "f(" + a + ")";
            }
            return def(ct.compute, std::string(rnd) + "(" + e + ")", in_body);
        }
        if (op == "is_finite") {
            const TensorType& x = g_.type(n->inputs[0]);
            std::string a = arg(0);
            return def("bool", dtype_is_float(x.dtype) ? "isfinite(" + a + ")" : "true", in_body);
        }
        if (op == "cast") {
            const TensorType& x = g_.type(n->inputs[0]);
            std::string a = arg(0), e;
            bool from_float = dtype_is_float(x.dtype);
            if (flt) {
                if (x.dtype == LB_BOOL) e = format("(%s ? (%s)1 : (%s)0)", a.c_str(), ct.compute, ct.compute);
                else e = format("%s((%s)%s)", rnd, ct.compute, a.c_str());
            } else if (t.dtype == LB_BOOL) {
                e = "(" + a + " != 0)";
            } else if (from_float) {
                static const char* lo[] = {"", "-128.0", "-32768.0", "-2147483648.0", "-9223372036854775808.0", "0.0", "0.0", "0.0", "0.0"};
                static const char* hi[] = {"", "127.0", "32767.0", "2147483647.0", "9223372036854775807.0", "255.0", "65535.0", "4294967295.0", "18446744073709551615.0"};
                static const char* tlo[] = {"", "-128", "-32768", "(-2147483647 - 1)", "(-9223372036854775807LL - 1)", "0", "0", "0u", "0ull"};
                static const char* thi[] = {"", "127", "32767", "2147483647", "9223372036854775807LL", "255", "65535", "4294967295u", "18446744073709551615ull"};
                e = format("sat_cast<%s>((double)%s, %s, %s, (%s)%s, (%s)%s)", ct.compute, a.c_str(), lo[t.dtype], hi[t.dtype], ct.compute, tlo[t.dtype], ct.compute, thi[t.dtype]);
            } else {
                e = format("(%s)%s", ct.compute, a.c_str());
            }
            return def(ct.compute, e, in_body);
        }
        if (op == "select") {
            return def(ct.compute, format("(%s ? %s : %s)", arg(0).c_str(), arg(1).c_str(), arg(2).c_str()), in_body);
        }
        if (op == "full") {
            const std::string& val = n->attr("fill_value");
            double x = val[0] == 'f' ? std::strtod(val.c_str() + 2, nullptr) : (double)std::stoll(val.substr(2));
            if (flt) return float_literal(host_round(x, t.dtype), t.dtype);
            if (t.dtype == LB_BOOL) return x != 0 ? "true" : "false";
            if (val[0] == 'f') fail(LB_ERR_UNSUPPORTED, "full: float fill value of an integer tensor");
            long long i = std::stoll(val.substr(2));
            return format("((%s)%lld%s)", ct.compute, i == INT64_MIN ? i + 1 : i, i == INT64_MIN ? "LL - 1" : "LL");
        }
        if (op == "iota") {
            const Comp& c = idx[n->integer("dimension")];
            std::string e = flt ? format("%s((%s)%s)", rnd, ct.compute, c.expr.c_str()) : format("(%s)%s", ct.compute, c.expr.c_str());
            return def(ct.compute, e, c.e_dep);
        }
        if (op == "broadcast_in_dim") {
            const TensorType& x = g_.type(n->inputs[0]);
            auto dims = n->ints("broadcast_dimensions");
            Index src(x.rank());
            for (int k = 0; k < x.rank(); k++) src[k] = x.shape[k] == 1 ? zero_comp() : idx[dims[k]];
            return gen(n->inputs[0], src, ph);
        }
        if (op == "transpose") {
            auto perm = n->ints("permutation");
            Index src(idx.size());
            for (size_t k = 0; k < perm.size(); k++) src[perm[k]] = idx[k];
            return gen(n->inputs[0], src, ph);
        }
        if (op == "reshape" || op == "device_wait" || op == "host_wait") {
            const TensorType& x = g_.type(n->inputs[0]);
            if (op != "reshape") return gen(n->inputs[0], idx, ph);
            // equal trailing dimensions pass through; the rest goes through the flat index
            int same = 0;
            while (same < x.rank() && same < t.rank() && x.shape[x.rank() - 1 - same] == t.shape[t.rank() - 1 - same]) same++;
            std::vector<int64_t> out_lead(t.shape.begin(), t.shape.end() - same), in_lead(x.shape.begin(), x.shape.end() - same);
            Index lead(idx.begin(), idx.end() - same);
            Index src = unravel(ravel(lead, out_lead), in_lead);
            src.insert(src.end(), idx.end() - same, idx.end());
            return gen(n->inputs[0], src, ph);
        }
        if (op == "slice") {
            auto start = n->ints("start_indices");
            Index src = idx;
            for (size_t k = 0; k < src.size(); k++) {
                if (start[k] == 0) continue;
                Comp& c = src[k];
                bool aligned = c.lane && start[k] % VEC_ == 0;
                if (c.lane && aligned) c.base = format("(%s + %lld)", c.base.c_str(), (long long)start[k]);
                else c.lane = false;
                c.expr = format("(%s + %lld)", c.expr.c_str(), (long long)start[k]);
                c.zero_known = 0;
            }
            return gen(n->inputs[0], src, ph);
        }
        if (op == "gather") {
            // out[..axis, i.., ..] = x[..axis, clamp(indices[i..]), ..]  (lumen/reference/mod.rs:731-749)
            const TensorType& x = g_.type(n->inputs[0]);
            const TensorType& ind = g_.type(n->inputs[1]);
            int axis = (int)n->integer("axis");
            Index sub(idx.begin() + axis, idx.begin() + axis + ind.rank());
            Comp picked;
            picked.e_dep = e_dep(sub);
            const bool pair_index = pairs_here(ph, picked.e_dep);
            std::string k = gen(n->inputs[1], sub, ph);
            if (pair_index) {
                ops.assign(1, k);
                k = "@0@";
            }
            picked.c_dep = c_dep(sub);
            picked.row_dep = true;
            picked.dyn = true;
            picked.expr = define(ph, "idx_t",
                                 format("(idx_t)imin<i64>(imax<i64>((i64)%s, 0), %lldLL)", k.c_str(),
                                        (long long)std::max<int64_t>(x.shape[axis] - 1, 0)),
                                 picked.e_dep, &ops, -1);
            if (pair_index) picked.expr = "LX(" + picked.expr + ")";
            Index src(idx.begin(), idx.begin() + axis);
            src.push_back(picked);
            src.insert(src.end(), idx.begin() + axis + ind.rank(), idx.end());
            return gen(n->inputs[0], src, ph);
        }
        if (op == "reduce_sum" || op == "reduce_max") return gen_reduce(*n, idx);
        fail(LB_ERR_UNSUPPORTED, "the fused kernel generator has no rule for primitive " + op);
    }

    std::string gen_reduce(const Node& n, const Index& idx) {
        if (mixed_ && !column_mode_ && behind_columns_.count(n.output))
            fail(LB_ERR_UNSUPPORTED, n.op + ": a column total read inside the rows it sums");
        if (column_mode_) {
            auto it = std::find(col_reduces_.begin(), col_reduces_.end(), n.output);
            if (it == col_reduces_.end()) fail(LB_ERR_UNSUPPORTED, n.op + ": mixed row and column reductions in one fusion");
            return format("tot%d[e]", (int)(it - col_reduces_.begin()));
        }
        if (e_dep(idx) || c_dep(idx))
            fail(LB_ERR_UNSUPPORTED, n.op + ": a row reduction read at a column-dependent index");
        std::string key = "red|" + key_of(n.output, idx);
        auto it = reduce_memo_.find(key);
        if (it != reduce_memo_.end()) return it->second;
        const TensorType& x = g_.type(n.inputs[0]);
        const TensorType& t = g_.type(n.output);
        auto axes = n.ints("axes");
        Index src = idx;
        if (axes.size() == 1) {
            src.push_back(col_comp());
        } else {
            std::vector<int64_t> tail(x.shape.end() - axes.size(), x.shape.end());
            Comp flat;
            flat.base = "c0";
            flat.expr = column();
            flat.lane = !shifted_;
            flat.e_dep = flat.c_dep = true;
            Index tail_idx = unravel(flat, tail);
            src.insert(src.end(), tail_idx.begin(), tail_idx.end());
        }
        Phase ph;
        ph.reduces = true;
        CType ct = ctype(t.dtype);
        ph.acc_type = ct.compute;
        ph.acc = fresh("acc");
        ph.result = fresh("red");
        bool sum = n.op == "reduce_sum";
        bool flt = dtype_is_float(t.dtype);
        if (sum) {
            ph.init = flt ? (t.dtype == LB_F64 ? "0.0" : "0.0f") : format("(%s)0", ct.compute);
            if (flt) ph.combine_a_b = t.dtype == LB_F64 ? "(%A + %B)" : format("%s(__fadd_rn(%%A, %%B))", rnd_fn(t.dtype));
            else ph.combine_a_b = format("(%s)((%s)%%A + (%s)%%B)", ct.compute, ct.unsigned_t, ct.unsigned_t);
        } else {
            if (flt) {
                ph.init = float_literal(-INFINITY, t.dtype);
                ph.combine_a_b = "fmax_nan(%A, %B)";
            } else {
                static const char* lowest[] = {"false", "(i8)-128", "(i16)-32768", "(-2147483647 - 1)", "(-9223372036854775807LL - 1)", "(u8)0", "(u16)0", "0u", "0ull"};
                ph.init = lowest[t.dtype];
                ph.combine_a_b = t.dtype == LB_BOOL ? "(%A || %B)" : format("imax<%s>(%%A, %%B)", ct.compute);
            }
        }
        std::string val = gen(n.inputs[0], src, ph);
        const bool pairs = adds_pairs(ph.combine_a_b, val);
        ph.sums = std::max(sums(sum && flt, pairs), pairs ? 2 : 1);
        const std::string which = shifted_ ? "e" : !pairs ? format("ch & %d", ph.sums - 1) : ph.sums == 2 ? "e & 1" : "(ch & 1) * 2 + (e & 1)";
        ph.body += accumulate(ph.sums == 1 ? ph.acc : ph.acc + "[" + which + "]", ph.combine_a_b, val);
        row_decls_ += format("%s %s;\n", ct.compute, ph.result.c_str());
        phases_.push_back(ph);
        reduce_memo_[key] = ph.result;
        return ph.result;
    }

    // A thread with many narrow vectors of a row keeps four sums: one chain over 16 elements, where wider vectors or more threads make it
    // four, had 1.35 times the error of a float32 sum over 3001. Shifted chunks, whose threads have as many elements, keep one a lane: which
    // elements those are follows from the row's distance to an aligned address, so that equal rows at different places (modulo eight), or of a
    // tensor that is not aligned, may differ in the last bits of a sum. The same call gives the same bits.
    // Where fewer threads walk a row than its sums were once dealt to, a thread's elements are dealt to as many sums as keep each no longer than
    // those threads' were in the mean (chain_), vector by vector: 88 elements of a float16 row of 8200 in one chain had 1.6 times the error of 16.
    // (Element by element, layer norm of 699 x 24000 float16 took 25.3 us instead of 17.8, softmax of 1699 x 9872 float32 27.6 instead of 25.4.) Pairs
    // that are added packed are two sums, of up to 44 elements: 2.9e-8 -> 3.3e-8 of a sum of 16384 exponentials, half a unit in its last place either way.
    int chain_ = 0;
    int sums(bool adds, bool pairs) const {
        if (shifted_) return VEC_;
        if (VEC_ <= 2) return NCH_ > 4 ? 4 : 1;
        int n = 1;
        while (adds && !pairs && chain_ && n < VEC_ && (NCH_ + n - 1) / n * VEC_ > chain_) n *= 2;
        return n;
    }

    // ---- emission ---------------------------------------------------------------------------------------
    std::string indent(const std::string& code, int n) {
        std::string pad(n, ' '), out;
        std::istringstream ss(code);
        for (std::string line; std::getline(ss, line);) out += pad + line + "\n";
        return out;
    }

    // `reads`: the kernel's parameters that it reads through
    static std::string wait_for_grid(int threads, const std::vector<std::string>& reads) {
        std::string s = "    const u32 tid = grid_wait();\n";
        for (const std::string& p : reads) s += "    " + p + " = behind_wait(" + p + ", tid);\n";
        return s + format("    __builtin_assume(tid < %du);\n", threads);
    }
    std::vector<std::string> input_names() const {
        std::vector<std::string> names;
        for (size_t i = 0; i < g_.inputs.size(); i++) names.push_back(format("in%d", (int)i));
        return names;
    }

    FusedKernel emit() {
        FusedKernel k;
        std::ostringstream s;
        std::vector<std::string> loops;
        for (const Phase& ph : phases_) loops.push_back(element_loops(ph));
        bool guard = C_ % ((int64_t)T_ * VEC_) != 0;
        s << "// generated by lumen_b200: fused row kernel over [" << R_ << ", " << C_ << "], " << T_
          << " threads per row, " << RPB_ << " rows per block, vectors of " << VEC_ << "\n";
        s << kPreamble;
        s << "typedef " << (wide_index_ ? "long long" : "int") << " idx_t;\n";
        s << "#define VEC " << VEC_ << "\n#define NCH " << NCH_ << "\n#define TPR " << T_ << "\n#define RPB " << RPB_ << "\n";
        s << "#define NCOLS " << C_ << "LL\n#define NROWS " << (multi_ ? std::string("group_rows") : std::to_string(R_) + "LL") << "\n";
        if (shifted_) {
            guard = true;
            s << "#define PERIOD " << period_ << "\n";
            s << "__device__ __forceinline__ idx_t column(idx_t c) { return c < 0 ? 0 : c < (idx_t)NCOLS ? c : (idx_t)(NCOLS - 1); }\n";
            s << "__device__ __forceinline__ bool in_row(idx_t c) { return c >= 0 && c < (idx_t)NCOLS; }\n";
        }
        s << "#define CHUNK_LOOP_BEGIN _Pragma(\"unroll\") for (int ch = 0; ch < NCH; ch++) { const idx_t c0 = (idx_t)(ch * TPR + lane_in_row) * VEC"
          << (shifted_ ? " - shift; const bool whole = c0 >= 0 && c0 + VEC <= (idx_t)NCOLS; " : "; ") << (guard ? "if (c0 < NCOLS) {" : "{") << "\n";
        s << "#define CHUNK_LOOP_END }}\n";
        // row reductions
        int width = std::min(T_, 32);
        s << "template <class A, class F> __device__ __forceinline__ A row_reduce(A v, F f, A identity, void* smem) {\n";
        s << "    #pragma unroll\n    for (int m = " << width / 2 << "; m >= 1; m >>= 1) v = f(v, shfl_xor_any<A>(v, m));\n";
        if (T_ > 32) {
            // the caller alternates between two areas of shared memory, so the next reduction's writes cannot overtake
            // this one's reads and one barrier is enough
            s << "    A* sm = (A*)smem; const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;\n";
            s << "    if (lane == 0) sm[warp] = v;\n    __syncthreads();\n";
            if (T_ <= 256) {  // every thread adds the warps' sums as the tree that the shuffles below are
                int warps = T_ / 32, p = 1;
                while (p < warps) p *= 2;
                s << "    A w[" << p << "];\n    #pragma unroll\n    for (int k = 0; k < " << p << "; k++) w[k] = k < " << warps << " ? sm[k] : identity;\n";
                s << "    #pragma unroll\n    for (int h = " << p / 2 << "; h >= 1; h /= 2) {\n        #pragma unroll\n        for (int k = 0; k < h; k++) w[k] = f(w[k], w[k + h]);\n    }\n    v = w[0];\n";
            } else {
                s << "    v = lane < " << T_ / 32 << " ? sm[lane] : identity;\n";
                s << "    #pragma unroll\n    for (int m = 16; m >= 1; m >>= 1) v = f(v, shfl_xor_any<A>(v, m));\n";
            }
        }
        s << "    return v;\n}\n";
        const char* restrict_kw = inplace_ ? "" : " __restrict__";
        const int n_ptrs = (int)(g_.inputs.size() + g_.outputs.size());
        if (multi_) {
            // Horizontal form (the reference's horizontal fusion of same-bodied kernels, lumen/graph_compiler/passes/
            // horizontal.rs:79): ONE launch applies the body to every group of a table passed by value - per group its
            // tensors' pointers and its row count. Only for bodies without reductions or row-constant operands.
            for (const Phase& ph : phases_)
                if (ph.reduces) fail(LB_ERR_UNSUPPORTED, "a horizontally fused kernel cannot hold a reduction");
            if (!kernel_cache_.empty() || !row_caches_.empty() || !row_decls_.empty())
                fail(LB_ERR_UNSUPPORTED, "a horizontally fused kernel takes full-shape operands and constants only");
            k.multi = true;
            k.multi_max_groups = std::max(1, (4000 - 24) / (8 * (n_ptrs + 1) + 4));  // the table fits the 4 KB parameter space
            s << "struct MultiTable { int n; u32 blocks; long long rows[" << k.multi_max_groups << "]; void* ptr[" << k.multi_max_groups << "]["
              << n_ptrs << "]; u32 first[" << k.multi_max_groups << "]; };\n";
            s << "extern \"C\" __global__ void __launch_bounds__(" << T_ * RPB_ << ") fused_kernel(const MultiTable table) {\n";
            s << wait_for_grid(T_ * RPB_, {});
            // The groups' row blocks form ONE sequence (`first`: each group's first place in it) dealt to the CTAs, of which there
            // are as many as blocks while they fit the GPU: a CTA looks its group up once and walks on. What bounds a small model's
            // update is latency: with every CTA visiting every group, as many CTAs as the largest group has blocks and a 64-bit
            // remainder per group, SGD over the 21 parameters of a 2-layer model took 16.7 us, now 4 (the whole step 310 -> 297).
            s << "  u32 group = 0;\n"
              << "  for (u32 below = table.n; below - group > 1;) { const u32 mid = (group + below) / 2; if (table.first[mid] <= blockIdx.x) group = mid; else below = mid; }\n";
            s << "  for (u32 block = blockIdx.x; block < table.blocks; block += gridDim.x) {\n";
            s << "    while (group + 1 < table.n && table.first[group + 1] <= block) group++;\n";
            s << "    const long long group_rows = table.rows[group];\n";
            for (size_t i = 0; i < g_.inputs.size(); i++) s << "    const void*" << restrict_kw << " in" << i << " = behind_wait(table.ptr[group][" << i << "], tid);\n";
            for (size_t i = 0; i < g_.outputs.size(); i++)
                s << "    void*" << restrict_kw << " out" << i << " = table.ptr[group][" << g_.inputs.size() + i << "];\n";
        } else {
            s << "extern \"C\" __global__ void __launch_bounds__(" << T_ * RPB_;
            if (mixed_ || shifted_) s << ", " << resident_;
            else if (per_sm_) s << ", " << per_sm_;
            s << ") fused_kernel(";
            for (size_t i = 0; i < g_.inputs.size(); i++) s << (i ? ", " : "") << "const void*" << restrict_kw << " in" << i;
            for (size_t i = 0; i < g_.outputs.size(); i++)
                s << ((i || !g_.inputs.empty()) ? ", " : "") << "void*" << restrict_kw << " out" << i;
            if (mixed_) s << ", void* __restrict__ scratch";
            s << ") {\n";
        }
        s << "    __shared__ unsigned long long red_smem[2][32];\n    int red_turn = 0;\n";
        if (!multi_) s << wait_for_grid(T_ * RPB_, input_names());
        s << "    const int lane_in_row = tid % TPR, row_in_block = tid / TPR;\n";
        // the row of a thread in row block %s
        auto row_of = [&](const std::string& rb) {
            return shifted_ ? "(" + rb + ") / PERIOD * (PERIOD * RPB) + row_in_block * PERIOD + (" + rb + ") % PERIOD" : "(" + rb + ") * RPB + row_in_block";
        };
        // (a row that stands in for one behind the last: loads go there and nothing else)
        auto stand_in = [&](const std::string& rb) { return shifted_ ? "(" + rb + ") % PERIOD" : std::string("(idx_t)(NROWS - 1)"); };
        if (shifted_)
            s << "    const idx_t row_blocks = (idx_t)((NROWS + PERIOD * RPB - 1) / (PERIOD * RPB)) * PERIOD;\n"
              << "    const int shift = (int)((blockIdx.x % PERIOD) * (u32)(NCOLS % VEC) % VEC);  // the grid is a multiple of PERIOD, or a block has one row block\n";
        else if (!multi_) s << "    const idx_t row_blocks = (idx_t)((NROWS + RPB - 1) / RPB);\n";
        s << indent(kernel_cache_, 4);
        for (size_t i = 0; i < col_reduces_.size(); i++) {
            const Node& n = *g_.node_of(col_reduces_[i]);
            std::string init, combine;
            reduce_ops(n, g_.type(n.output), &init, &combine);
            s << "    " << ctype(g_.type(n.output).dtype).compute << " cacc" << i << "[NCH][VEC];\n";
            s << "    _Pragma(\"unroll\") for (int ch = 0; ch < NCH; ch++) { _Pragma(\"unroll\") for (int e = 0; e < VEC; e++) cacc" << i << "[ch][e] = " << init << "; }\n";
        }
        // Rows cached in registers are loaded one row block ahead (while the current block's phases compute), when that
        // costs at most 64 bytes of registers per thread: a block's phases are a serial chain behind its loads.
        int cached_bytes = 0;
        for (const RowCache& c : row_caches_) cached_bytes += c.bytes;
        const bool prefetch = !inplace_ && !row_caches_.empty() && cached_bytes <= 64;
        std::string next_loads;
        if (prefetch) {
            for (const RowCache& c : row_caches_) {
                s << "    __align__(16) " << c.type << " " << c.buf << "_nx[NCH][VEC];\n";
                next_loads += c.load;
            }
            s << "    if ((idx_t)blockIdx.x < row_blocks) {\n        idx_t r = " << row_of("(idx_t)blockIdx.x") << ";\n"
              << "        if (r >= NROWS) r = " << stand_in("(idx_t)blockIdx.x") << ";\n" << indent(next_loads, 8) << "    }\n";
        }
        if (multi_) s << "    {\n        const idx_t rb = block - table.first[group];\n";
        else s << "    for (idx_t rb = blockIdx.x; rb < row_blocks; rb += gridDim.x) {\n";
        s << "        idx_t r = " << row_of("rb") << ";\n";
        s << "        const bool active = r < NROWS;\n";
        s << "        if (!active) r = " << stand_in("rb") << ";\n";
        s << indent(row_decls_, 8);
        if (prefetch) {
            for (const RowCache& c : row_caches_) {
                s << "        __align__(16) " << c.type << " " << c.buf << "[NCH][VEC];\n";
                s << "        _Pragma(\"unroll\") for (int ch = 0; ch < NCH; ch++) { _Pragma(\"unroll\") for (int e = 0; e < VEC; e++) " << c.buf
                  << "[ch][e] = " << c.buf << "_nx[ch][e]; }\n";
            }
            s << "        if (rb + (idx_t)gridDim.x < row_blocks) {\n            idx_t r = " << row_of("rb + (idx_t)gridDim.x") << ";\n"
              << "            if (r >= NROWS) r = " << stand_in("rb + (idx_t)gridDim.x") << ";\n" << indent(next_loads, 12) << "        }\n";
        } else {
            s << indent(row_cache_, 8);
        }
        for (size_t at = 0; at < phases_.size(); at++) {
            const Phase& ph = phases_[at];
            s << "        {\n";
            if (ph.reduces && ph.sums > 1) {
                s << "            " << ph.acc_type << " " << ph.acc << "[" << ph.sums << "] = {" << ph.init;
                for (int n = 1; n < ph.sums; n++) s << ", " << ph.init;
                s << "};\n";
            } else if (ph.reduces) s << "            " << ph.acc_type << " " << ph.acc << " = " << ph.init << ";\n";
            if (ph.chunked) {
                s << "            CHUNK_LOOP_BEGIN\n";
                s << indent(ph.pre, 16);
                s << indent(loops[at], 16);
                s << indent(ph.post, 16);
                s << "            CHUNK_LOOP_END\n";
            } else {
                s << indent(ph.pre, 12);
            }
            if (ph.reduces) {
                std::string sum = ph.acc;
                std::vector<std::string> tree;
                for (int n = 0; ph.sums > 1 && n < ph.sums; n++) tree.push_back(format("%s[%d]", ph.acc.c_str(), n));
                for (; tree.size() > 1; tree.resize(tree.size() / 2))
                    for (size_t n = 0; n < tree.size() / 2; n++) tree[n] = subst(ph.combine_a_b, tree[2 * n], tree[2 * n + 1]);
                if (!tree.empty()) sum = tree[0];
                s << "            " << ph.result << " = row_reduce<" << ph.acc_type << ">(" << sum << ", [](" << ph.acc_type
                  << " a, " << ph.acc_type << " b) { return " << subst(ph.combine_a_b, "a", "b") << "; }, (" << ph.acc_type
                  << ")" << ph.init << ", red_smem[red_turn ^= 1]);\n";
            }
            s << "        }\n";
        }
        s << (multi_ ? "    }\n  }\n" : "    }\n");
        if (mixed_) {
            // enough CTAs to keep several rows in flight on every SM; each leaves one slice of partial sums per column
            const int64_t row_blocks = std::max<int64_t>((R_ + RPB_ - 1) / RPB_, 1);
            k.two_pass = true;
            // (but no more than 592 while they have less than four row blocks each: every one leaves a slice that the totals read. 1024 x 512
            // bfloat16, us, 1024 slices -> 592: 9.9 -> 8.4, 2048 x 512 12.2 -> 10)
            k.col_blocks = std::min(std::min<int64_t>(row_blocks, 148LL * resident_), std::max<int64_t>(592, row_blocks / 4));
            k.slices = 1;
            std::vector<size_t> offsets;
            size_t scratch = 0;
            if (RPB_ > 1) s << "    __shared__ __align__(16) char shared[NCOLS * 8];\n";
            for (size_t i = 0; i < col_reduces_.size(); i++) {
                const Node& n = *g_.node_of(col_reduces_[i]);
                const TensorType& t = g_.type(n.output);
                const std::string type = ctype(t.dtype).compute;
                const int width = type == "float" ? 4 : type == "double" ? 8 : dtype_size(t.dtype);
                std::string init, combine;
                reduce_ops(n, t, &init, &combine);
                s << "    {\n        " << type << "* part = (" << type << "*)((char*)scratch + " << scratch << ") + (idx_t)blockIdx.x * NCOLS;\n";
                if (RPB_ > 1) {  // the rows of a warp as a tree, then the warps in order, through shared memory
                    const std::string acc = format("cacc%d[ch][e]", (int)i), sum = format("csum%d[c0 + e]", (int)i);
                    s << "        " << type << "* csum" << i << " = (" << type << "*)shared;\n";
                    s << "        _Pragma(\"unroll\") for (int ch = 0; ch < NCH; ch++) { _Pragma(\"unroll\") for (int e = 0; e < VEC; e++) { _Pragma(\"unroll\") for (int m = TPR; m < 32; m *= 2) "
                      << acc << " = " << subst(combine, acc, format("shfl_xor_any<%s>(%s, m)", type.c_str(), acc.c_str())) << "; } }\n";
                    s << "        for (int y = 0; y < TPR * RPB / 32; y++) {\n            if (threadIdx.x / 32 == y && threadIdx.x % 32 < TPR) { CHUNK_LOOP_BEGIN _Pragma(\"unroll\") for (int e = 0; e < VEC; e++) "
                      << sum << " = y ? " << subst(combine, sum, acc) << " : " << acc << "; CHUNK_LOOP_END }\n            __syncthreads();\n        }\n";
                    s << "        for (int c = threadIdx.x; c < NCOLS; c += TPR * RPB) part[c] = csum" << i << "[c];\n        __syncthreads();\n    }\n";
                } else {
                    s << "        CHUNK_LOOP_BEGIN _Pragma(\"unroll\") for (int e = 0; e < VEC; e++) part[c0 + e] = cacc" << i << "[ch][e]; CHUNK_LOOP_END\n    }\n";
                }
                offsets.push_back(scratch);
                scratch = (scratch + (size_t)k.col_blocks * C_ * width + 255) & ~(size_t)255;
            }
            s << "}\n#define SLICES " << k.col_blocks << "\n";
            std::string sig;
            for (size_t i = 0; i < g_.inputs.size(); i++) sig += format("const void* __restrict__ in%d, ", (int)i);
            for (size_t i = 0; i < g_.outputs.size(); i++) sig += format("void* __restrict__ out%d, ", (int)i);
            k.vec = VEC_;
            emit_finalize(s, sig + "void* __restrict__ scratch", offsets, column_outputs_, k);
            k.scratch_bytes = scratch;
        } else {
            s << "}\n";
            k.vec = VEC_, k.shifted = shifted_;
        }
        k.source = s.str();
        k.rows = R_;
        k.cols = C_;
        k.threads = T_ * RPB_;
        k.rows_per_block = RPB_;
        k.row_period = period_;
        if (shifted_) k.per_sm = resident_;
        else k.per_sm = per_sm_;
        k.n_inputs = (int)g_.inputs.size();
        k.n_outputs = (int)g_.outputs.size();
        for (int v : g_.inputs) k.types.push_back(g_.type(v));
        for (int v : g_.outputs) k.types.push_back(g_.type(v));
        return k;
    }

  public:
    void set_multi_phase(bool v) { multi_phase_hint_ = v; }
    // ---- column mode: reductions over the leading axes ------------------------------------------------------
    // Pass 1 (fused_kernel): grid (column blocks, row slices); a thread owns VEC columns and adds its slice's rows
    // in order. Pass 2 (fused_finalize): a thread adds the slices' partial sums in order and applies the epilogue.
    // The order of every sum is fixed, so results are bit-reproducible.
    static bool leading_axes(const Node& n, const TensorType& x, int* lead) {
        auto axes = n.ints("axes");
        std::sort(axes.begin(), axes.end());
        if (axes.empty() || (int)axes.size() >= x.rank()) return false;
        for (size_t k = 0; k < axes.size(); k++)
            if (axes[k] != (int64_t)k) return false;
        *lead = (int)axes.size();
        return true;
    }

    FusedKernel run_columns() {
        column_mode_ = true;
        const TensorType* space = nullptr;
        for (const Node& n : g_.nodes) {
            if (n.op != "reduce_sum" && n.op != "reduce_max") continue;
            const TensorType& x = g_.type(n.inputs[0]);
            int lead = 0;
            if (!leading_axes(n, x, &lead)) fail(LB_ERR_UNSUPPORTED, "mixed row and column reductions in one fusion");
            int64_t r = 1;
            for (int d = 0; d < lead; d++) r *= x.shape[d];
            int64_t c = x.numel() / std::max<int64_t>(r, 1);
            if (space && (r != R_ || c != C_)) fail(LB_ERR_UNSUPPORTED, "column reductions over different shapes in one fusion");
            space = &x, R_ = r, C_ = r ? c : 0, lead_rank_ = lead;
            col_reduces_.push_back(n.output);
        }
        has_reduce_ = true;
        int min_size = 8;
        for (int v : g_.inputs)
            if (g_.type(v).numel() == R_ * C_) min_size = std::min(min_size, dtype_size(g_.type(v).dtype));
        VEC_ = std::min(8, 16 / min_size);
        while (VEC_ > 1 && (C_ % VEC_ != 0 || space->shape.back() % VEC_ != 0)) VEC_ /= 2;
        wide_index_ = R_ * C_ >= (1LL << 31) - 4096;
        pair_ = VEC_ >= 2 && computes_bf16();
        // both passes: 256 threads = 32 column lanes (VEC columns each) x 8 row lanes (pass 2: slice lanes)
        const int threads = 256, col_lanes = 32, row_lanes = 8;
        int64_t col_blocks = std::max<int64_t>((C_ + (int64_t)col_lanes * VEC_ - 1) / ((int64_t)col_lanes * VEC_), 1);
        // enough slices to fill the GPU a few times over, each at least 64 rows long
        int64_t slices = std::min<int64_t>(std::max<int64_t>(1, (148 * 4 + col_blocks - 1) / col_blocks), std::max<int64_t>(R_ / 64, 1));
        int64_t rows_per_slice = (R_ + slices - 1) / std::max<int64_t>(slices, 1);
        slices = rows_per_slice ? (R_ + rows_per_slice - 1) / rows_per_slice : 1;

        std::vector<int64_t> lead_shape(space->shape.begin(), space->shape.begin() + lead_rank_);
        std::vector<int64_t> trail_shape(space->shape.begin() + lead_rank_, space->shape.end());
        Comp flat_c;
        flat_c.base = "c0", flat_c.expr = "(c0 + e)";
        flat_c.lane = flat_c.e_dep = flat_c.c_dep = true;

        // pass 1
        Phase part;
        std::ostringstream decl, store;
        size_t scratch = 0;
        int widest = 1;  // all reductions use one area of shared memory in turn: any number of them fits
        std::vector<size_t> offsets;
        for (size_t k = 0; k < col_reduces_.size(); k++) {
            const Node& n = *g_.node_of(col_reduces_[k]);
            const TensorType& t = g_.type(n.output);
            CType ct = ctype(t.dtype);
            Index idx = unravel(row_comp(), lead_shape);
            Index tail = unravel(flat_c, trail_shape);
            idx.insert(idx.end(), tail.begin(), tail.end());
            bool prev = column_mode_;
            std::string val = gen(n.inputs[0], idx, part);
            column_mode_ = prev;
            std::string init, combine;
            reduce_ops(n, t, &init, &combine);
            decl << ct.compute << " acc" << k << "[VEC];\n#pragma unroll\nfor (int e = 0; e < VEC; e++) acc" << k << "[e] = " << init << ";\n";
            part.body += accumulate(format("acc%d[e]", (int)k), combine, val);
            offsets.push_back(scratch);
            int width = std::string(ct.compute) == "double" || std::string(ct.compute) == "i64" || std::string(ct.compute) == "u64" ? 8
                        : (std::string(ct.compute) == "float" || std::string(ct.compute) == "i32" || std::string(ct.compute) == "u32") ? 4
                        : dtype_size(t.dtype);
            // the 8 row lanes of a column are combined in lane order through shared memory, then lane 0 stores the slice's partial
            widest = std::max(widest, width);
            if (k) store << "__syncthreads();\n";
            store << "auto red" << k << " = (" << ct.compute << "(*)[" << col_lanes << " * VEC])shared;\n";
            store << "#pragma unroll\nfor (int e = 0; e < VEC; e++) red" << k << "[row_lane][col_lane * VEC + e] = acc" << k << "[e];\n__syncthreads();\n";
            store << "if (row_lane == 0 && in_range) {\n#pragma unroll\n    for (int e = 0; e < VEC; e++) {\n        " << ct.compute << " t = acc" << k
                  << "[e];\n        for (int y = 1; y < " << row_lanes << "; y++) t = " << subst(combine, "t", format("red%d[y][col_lane * VEC + e]", (int)k))
                  << ";\n        ((" << ct.compute << "*)((char*)scratch + " << scratch << "))[(idx_t)blockIdx.y * NCOLS + c0 + e] = t;\n    }\n}\n";
            scratch += (size_t)slices * C_ * width;
            scratch = (scratch + 255) & ~(size_t)255;
        }
        std::ostringstream s;
        s << "// generated by lumen_b200: column reduction over [" << R_ << " rows, " << C_ << " columns], " << slices << " row slices\n";
        s << kPreamble;
        s << "typedef " << (wide_index_ ? "long long" : "int") << " idx_t;\n";
        s << "#define VEC " << VEC_ << "\n#define NCOLS " << C_ << "LL\n#define NROWS " << R_ << "LL\n#define SLICES " << slices
          << "\n#define ROWS_PER_SLICE " << rows_per_slice << "LL\n";
        std::string sig;
        for (size_t i = 0; i < g_.inputs.size(); i++) sig += format("const void* __restrict__ in%d, ", (int)i);
        for (size_t i = 0; i < g_.outputs.size(); i++) sig += format("void* __restrict__ out%d, ", (int)i);
        sig += "void* __restrict__ scratch";
        s << "extern \"C\" __global__ void __launch_bounds__(" << threads << ") fused_kernel(" << sig << ") {\n";
        s << wait_for_grid(threads, input_names());
        s << "    const int col_lane = tid & " << col_lanes - 1 << ", row_lane = tid >> 5;\n";
        s << "    const idx_t c0 = ((idx_t)blockIdx.x * " << col_lanes << " + col_lane) * VEC;\n    const bool in_range = c0 < NCOLS;\n";
        s << "    __shared__ __align__(16) char shared[" << row_lanes * col_lanes << " * VEC * " << widest << "];\n";
        s << indent(decl.str(), 4);
        s << "    const idx_t r_end = in_range ? (idx_t)(((idx_t)blockIdx.y + 1) * ROWS_PER_SLICE < NROWS ? ((idx_t)blockIdx.y + 1) * ROWS_PER_SLICE : NROWS) : 0;\n";
        s << "    for (idx_t r = (idx_t)blockIdx.y * ROWS_PER_SLICE + row_lane; r < r_end; r += " << row_lanes << ") {\n";
        s << indent(part.pre, 8);
        s << "        #pragma unroll\n        for (int e = 0; e < VEC; e += " << (pair_ ? 2 : 1) << ") {\n" << indent(part.body, 12) << "        }\n    }\n";
        s << indent(store.str(), 4);
        s << "}\n";
        FusedKernel k;
        std::vector<int> outputs(g_.outputs.size());
        for (size_t i = 0; i < outputs.size(); i++) outputs[i] = (int)i;
        k.slices = (int)slices;
        emit_finalize(s, sig, offsets, outputs, k);
        k.source = s.str();
        k.rows = R_, k.cols = C_, k.threads = threads, k.rows_per_block = 1, k.vec = VEC_;
        k.n_inputs = (int)g_.inputs.size(), k.n_outputs = (int)g_.outputs.size();
        for (int v : g_.inputs) k.types.push_back(g_.type(v));
        for (int v : g_.outputs) k.types.push_back(g_.type(v));
        k.two_pass = true;
        k.slices = (int)slices;
        k.col_blocks = col_blocks;
        k.scratch_bytes = scratch;
        return k;
    }

    // The second kernel of a column reduction: adds the slices' partial sums and applies the epilogue. A block takes 32
    // lanes of two columns and one (up to eight slices), eight or 32 slice lanes: few columns and slices per thread, so that the chains of loads stay
    // short (1184 slices of 1024 columns took 19 us with eight slice lanes). Many slices of few columns take 128 slice lanes, on eight
    // column lanes: four times the blocks, and a thread's chain of loads a quarter (a residual layer norm of 8192 x 1024 with its
    // backward, whose totals are 592 slices of 1024 columns, 36.1 -> 33.5 us). Where the line lies, by the time of a whole kernel pair with
    // 128 lanes over that with 32: 1184 slices of 512 columns 0.60 - 0.73, 592 of 1024 0.71 - 0.88, 296 of 2048 0.90 - 0.98, 260 of 500
    // to 2048 0.85 - 0.94, 296 of 3072 1.00; 296 of 2049, one column a thread, 1.00 - 1.01; 148 of 6144 1.02 - 1.21. Fewer slices were
    // measured faster too (200 of 500 to 2048 0.89 - 0.95, 128 of up to 256 0.93) down to 64 (1.01), but are left as they are.
    void emit_finalize(std::ostringstream& s, const std::string& sig, const std::vector<size_t>& offsets, const std::vector<int>& outputs, FusedKernel& k) {
        column_mode_ = true;
        VEC_ = std::min(VEC_, 2);
        pair_ = VEC_ >= 2 && computes_bf16();
        const int64_t slices = k.slices * k.col_blocks;
        const bool many = slices > 256 && C_ <= 64LL * VEC_ * 32;
        const int col_lanes = many ? 8 : 32, row_lanes = many ? 128 : slices > 64 ? 32 : slices > 8 ? 8 : 1, threads = col_lanes * row_lanes;
        const int warp_lanes = std::min(row_lanes, 32);  // lanes of a column that are added by shuffles
        Comp flat_c;
        flat_c.base = "c0", flat_c.expr = "(c0 + e)";
        flat_c.lane = flat_c.e_dep = flat_c.c_dep = true;
        Phase fin;
        std::ostringstream totals;
        int widest = 1;  // of the compute types; one area of shared memory serves the reductions in turn
        // Slice lane y adds slices y, y + (lanes), ... in four sums in turn, whose loads are in flight together; the sums and then the
        // lanes are combined as trees (one chain a lane and the lanes in order had up to 1.6 times the error of a float32 sum over
        // 1184 slices). For the second tree a column's lanes lie side by side in a warp (rows padded by one against bank
        // conflicts), for as many reductions at once as 40 KB of shared memory hold.
        for (int v : col_reduces_) {
            const int dtype = g_.type(v).dtype;
            widest = std::max(widest, dtype == LB_BF16 || dtype == LB_F16 ? 4 : dtype_size(dtype));
        }
        const int lane_bytes = row_lanes * (col_lanes * VEC_ + 1) * widest, sum_bytes = col_lanes * VEC_ * widest;
        const size_t batch = std::min<size_t>(col_reduces_.size(), std::max(1, 40 * 1024 / (lane_bytes + sum_bytes)));
        for (size_t k0 = 0; k0 < col_reduces_.size(); k0 += batch) {
            std::ostringstream trees, reads;
            for (size_t k = k0; k < std::min(k0 + batch, col_reduces_.size()); k++) {
                const Node& n = *g_.node_of(col_reduces_[k]);
                const TensorType& t = g_.type(n.output);
                const std::string type = ctype(t.dtype).compute, run = format("run%d", (int)k), tot = format("tot%d", (int)k);
                std::string init, combine;
                reduce_ops(n, t, &init, &combine);
                auto each = [&](const std::string& body) { return "_Pragma(\"unroll\") for (int e = 0; e < VEC; e++) { " + body + " }"; };
                auto add = [&](const std::string& to, const std::string& x) { return to + " = " + subst(combine, to, x) + ";"; };
                const std::string from = format("((const %s*)((const char*)scratch + %zu))[(idx_t)(s + u * %d) * NCOLS + c0 + e]", type.c_str(), offsets[k], row_lanes);
                const std::string unrolled = "_Pragma(\"unroll\") for (int u = 0; u < %d; u++) ", four = format(unrolled.c_str(), 4), three = format(unrolled.c_str(), 3);
                const std::string lanes = format("auto lanes = (%s(*)[%d * VEC + 1])(shared + %zu);\n    ", type.c_str(), col_lanes, (k - k0) * lane_bytes);
                const size_t sums_at = batch * lane_bytes + (k - k0) * sum_bytes;
                // a lane's slices: four at once, then the up to three that are left, then the four sums
                totals << type << " " << tot << "[VEC];\n{\n"
                       << "    " << type << " " << run << "[4][VEC];\n"
                       << "    " << four << each(run + "[u][e] = " + init + ";") << "\n"
                       << "    if (in_range) {\n"
                       << "        int s = row_lane;\n"
                       << "        #pragma unroll 2\n"
                       << "        for (; s + " << 3 * row_lanes << " < SLICES; s += " << 4 * row_lanes << ") {\n"
                       << "            " << type << " pv[4][VEC];\n"
                       << "            " << four << each("pv[u][e] = " + from + ";") << "\n"
                       << "            " << four << each(add(run + "[u][e]", "pv[u][e]")) << "\n"
                       << "        }\n"
                       << "        " << three << "if (s + u * " << row_lanes << " < SLICES) " << each("const " + type + " pv = " + from + "; " + add(run + "[u][e]", "pv")) << "\n"
                       << "    }\n"
                       << "    " << each(add(run + "[0][e]", run + "[1][e]") + " " + add(run + "[2][e]", run + "[3][e]") + " " + tot + "[e] = " + subst(combine, run + "[0][e]", run + "[2][e]") + ";") << "\n    ";
                if (row_lanes > 1) totals << lanes << each("lanes[row_lane][col_lane * VEC + e] = " + tot + "[e];") << "\n";
                totals << "}\n";
                // the lanes of a column, which a warp takes side by side: 128 are four to a thread of the first `col_lanes` warps
                std::string tree = type + " v = lanes[lane][col * VEC + e]; ";
                if (many)
                    tree += type + " v1 = lanes[lane + 32][col * VEC + e], v2 = lanes[lane + 64][col * VEC + e]; " + add("v", "v1") +
                            " v1 = lanes[lane + 96][col * VEC + e]; " + add("v2", "v1") + " " + add("v", "v2") + " ";
                tree += format("_Pragma(\"unroll\") for (int m = %d; m >= 1; m /= 2) ", warp_lanes / 2) + add("v", "shfl_xor_any<" + type + ">(v, m)") +
                        " if (lane == 0) sums[col * VEC + e] = v;";
                trees << "{\n    " << lanes << type << "* sums = (" << type << "*)(shared + " << sums_at << ");\n"
                      << "    const int lane = threadIdx.x % " << warp_lanes << ", col = threadIdx.x / " << warp_lanes << ";\n"
                      << "    " << (many ? format("if (col < %d) ", col_lanes) : "") << each(tree) << "\n}\n";
                reads << each(tot + "[e] = ((const " + type + "*)(shared + " + std::to_string(sums_at) + "))[col_lane * VEC + e];") << "\n";
            }
            if (row_lanes > 1) totals << "__syncthreads();\n" << trees.str() << "__syncthreads();\n" << reads.str();
            // (the next batch writes `lanes`, which were read before the last barrier; its trees write `sums` after another one)
        }
        const size_t shared_bytes = row_lanes == 1 ? 16 : batch * (lane_bytes + sum_bytes);
        for (int o : outputs) {
            const TensorType& t = g_.type(g_.outputs[o]);
            if (t.numel() != C_) fail(LB_ERR_UNSUPPORTED, format("column-reduction fusion output %s does not have %lld elements", t.str().c_str(), (long long)C_));
            Index idx = unravel(flat_c, t.shape);
            std::string val = gen(g_.outputs[o], idx, fin);
            CType ct = ctype(t.dtype);
            fin.pre += format("__align__(16) %s ob%d[VEC];\n", ct.memory, o);
            fin.body += store_element(format("ob%d", o), t.dtype, val);
            fin.post += format("stv<%s, VEC>((%s*)out%d + c0, ob%d);\n", ct.memory, ct.memory, o, o);
        }
        s << "#undef VEC\n#define VEC " << VEC_ << "\n";
        s << "extern \"C\" __global__ void __launch_bounds__(" << threads << ") fused_finalize(" << sig << ") {\n";
        std::vector<std::string> reads = input_names();
        reads.push_back("scratch");
        s << wait_for_grid(threads, reads);
        s << "    const int col_lane = tid & " << col_lanes - 1 << ", row_lane = tid / " << col_lanes << ";\n";
        s << "    const idx_t c0 = ((idx_t)blockIdx.x * " << col_lanes << " + col_lane) * VEC;\n    const bool in_range = c0 < NCOLS;\n";
        s << "    __shared__ __align__(16) char shared[" << shared_bytes << "];\n";
        s << indent(totals.str(), 4);
        s << "    if (row_lane != 0 || !in_range) return;\n";
        s << indent(fin.pre, 4);
        s << "    #pragma unroll\n    for (int e = 0; e < VEC; e += " << (pair_ ? 2 : 1) << ") {\n" << indent(fin.body, 8) << "    }\n";
        s << indent(fin.post, 4);
        s << "}\n";
        k.fin_threads = threads;
        k.fin_blocks = std::max<int64_t>((C_ + (int64_t)col_lanes * VEC_ - 1) / ((int64_t)col_lanes * VEC_), 1);
    }

    // identity and combine format of a reduction node with result type `t`
    void reduce_ops(const Node& n, const TensorType& t, std::string* init, std::string* combine) {
        CType ct = ctype(t.dtype);
        bool sum = n.op == "reduce_sum", flt = dtype_is_float(t.dtype);
        if (sum) {
            *init = flt ? (t.dtype == LB_F64 ? "0.0" : "0.0f") : format("(%s)0", ct.compute);
            if (flt) *combine = t.dtype == LB_F64 ? "(%A + %B)" : format("%s(__fadd_rn(%%A, %%B))", rnd_fn(t.dtype));
            else *combine = format("(%s)((%s)%%A + (%s)%%B)", ct.compute, ct.unsigned_t, ct.unsigned_t);
        } else if (flt) {
            *init = float_literal(-INFINITY, t.dtype);
            *combine = "fmax_nan(%A, %B)";
        } else {
            static const char* lowest[] = {"false", "(i8)-128", "(i16)-32768", "(-2147483647 - 1)", "(-9223372036854775807LL - 1)", "(u8)0", "(u16)0", "0u", "0ull"};
            *init = lowest[t.dtype];
            *combine = t.dtype == LB_BOOL ? "(%A || %B)" : format("imax<%s>(%%A, %%B)", ct.compute);
        }
    }

    static bool wants_columns(const Graph& g) {
        bool any = false;
        for (const Node& n : g.nodes) {
            if (n.op != "reduce_sum" && n.op != "reduce_max") continue;
            int lead;
            if (!leading_axes(n, g.type(n.inputs[0]), &lead)) return false;
            any = true;
        }
        return any;
    }
    static bool some_columns(const Graph& g) {
        int lead;
        for (const Node& n : g.nodes)
            if ((n.op == "reduce_sum" || n.op == "reduce_max") && leading_axes(n, g.type(n.inputs[0]), &lead)) return true;
        return false;
    }
    // whether an output is not computed from a column total
    static bool leaves_rows(const Graph& g) {
        std::set<int> behind;
        for (const Node& n : g.nodes) {
            bool in = n.op == "reduce_sum" || n.op == "reduce_max";
            for (int v : n.inputs) in |= behind.count(v) != 0;
            if (in) behind.insert(n.output);
        }
        for (int v : g.outputs)
            if (!behind.count(v)) return true;
        return false;
    }
    void set_inplace(bool v) { inplace_ = v; }
    void set_multi(bool v) { multi_ = v; }
    void set_mixed(bool v) { mixed_ = v; }
    void set_shifts(bool v) { shifts_ = v; }
    void set_sixteen_warps(bool v) { sixteen_warps_ = v; }

};

}  // namespace

static FusedKernel generate(const Module& module, bool shifts) {
    const Graph& g = module.main();
    int reduces = 0;
    for (const Node& n : g.nodes)
        if (n.op == "reduce_sum" || n.op == "reduce_max") reduces++;
    Generator gen(module, g);
    gen.set_inplace(module.options.count("inplace") != 0);
    gen.set_multi(module.options.count("multi") != 0);
    gen.set_sixteen_warps(module.options.count("sixteen_warps") != 0);
    if (module.options.count("multi") && (reduces || Generator::wants_columns(g)))
        fail(LB_ERR_UNSUPPORTED, "option multi: a horizontally fused kernel cannot hold a reduction");
    if (Generator::wants_columns(g) && !Generator::leaves_rows(g)) return gen.run_columns();
    if (Generator::some_columns(g) && !module.options.count("inplace")) gen.set_mixed(true);
    // With a reduction followed by further use of the row, inputs are kept in registers across phases.
    gen.set_multi_phase(reduces >= 1);
    gen.set_shifts(shifts);
    return gen.run();
}

FusedKernel generate_fused(const Module& module) {
    FusedKernel k = generate(module, true);
    if (!k.shifted) return k;
    k.unaligned = std::make_shared<FusedKernel>(generate(module, false));
    k.scratch_bytes = std::max(k.scratch_bytes, k.unaligned->scratch_bytes);
    return k;
}

}  // namespace lb
