// Error-bounded quantiser, dequantiser and the dense q.k baseline.
//
// Follows utils/compute.py:93-106 (quant) as torch evaluates it on fp16 tensors: every
// elementwise op widens to fp32, computes, and rounds to nearest-even back to fp16; the
// Python scalar `rel` stays fp32.  Explicit round-to-nearest intrinsics are used so that no
// contraction or fast-math rewrite can change a bit.
#include <string.h>

#include <algorithm>

#include "kvc_common.cuh"

namespace {

struct UnitParam { float sf; float mi; float rcp; };   // scale, min_int and 1/scale as floats

__device__ __forceinline__ UnitParam unit_param(float mn, float mx, float rel, __half *scale_out, int *flags) {
    __half range = __float2half_rn(__fsub_rn(mx, mn));
    __half sc = __float2half_rn(__fmul_rn(__half2float(range), rel));
    UnitParam p;
    p.sf = __half2float(sc);
    p.rcp = 0.0f;
    if (p.sf == 0.0f || p.sf != p.sf) { p.mi = 0.0f; *flags |= KVC_FLAG_ZERO_SCALE; }
    else { p.mi = rintf(__half2float(__float2half_rn(__fdiv_rn(mn, p.sf)))); p.rcp = __frcp_rn(p.sf); }
    *scale_out = sc;
    return p;
}

__device__ __forceinline__ void store_min(void *min_int, int min_bytes, long long u, float mi, int *flags) {
    int v = (int)mi;
    if (min_bytes == 1) {
        if (v < -128 || v > 127) *flags |= KVC_FLAG_MIN_OVERFLOW;
        reinterpret_cast<int8_t *>(min_int)[u] = (int8_t)v;      // wraps like the reference's .to(int8)
    } else {
        if (v < -32768 || v > 32767) *flags |= KVC_FLAG_MIN_OVERFLOW;
        reinterpret_cast<int16_t *>(min_int)[u] = (int16_t)v;
    }
}

// fp16(x / scale) without the full IEEE division: q1 = x*r corrected once by the exact residual is within
// 2^-24 (relative) of the true quotient t.  x and scale carry 11 significant bits, so t is at least
// 2^-23 (relative) away from every midpoint between two fp16 values (t = m would need m*scale = x with a
// 12-bit m); hence q1, the correctly rounded fp32 quotient and t all round to the same fp16 value.
// rint(v) for |v| < 2^22 without the conversion pipe: adding 1.5 * 2^23 rounds to an integer (to nearest
// even, the mode rintf uses) and leaves that integer in the low mantissa bits.
#define KVC_RINT_MAGIC 12582912.0f
__device__ __forceinline__ uint32_t quant_one(__half x, const UnitParam &p, int *flags) {
    if (p.sf == 0.0f || p.sf != p.sf) return 0u;
    const float xf = __half2float(x);
    const float q0 = __fmul_rn(xf, p.rcp);
    const float q1 = __fmaf_rn(__fmaf_rn(-q0, p.sf, xf), p.rcp, q0);
    const float qh = __half2float(__float2half_rn(q1));                      // |qh| <= 65504 (or inf)
    const float q = __fsub_rn(__fadd_rn(qh, KVC_RINT_MAGIC), KVC_RINT_MAGIC);  // = rintf(qh) for finite qh
    const float d = __fsub_rn(q, p.mi);
    if (d >= 0.0f && d <= 255.0f)            // an integer that fp16 holds exactly: the code, read from the mantissa
        return (uint32_t)__float_as_int(__fadd_rn(d, KVC_RINT_MAGIC)) & 0xffu;
    // out of range (or not finite): follow the fp16 arithmetic to the end, as the reference's tensors do
    const float qs = rintf(qh);
    const float c = __half2float(__float2half_rn(__fsub_rn(qs, p.mi)));
    if (!(c >= 0.0f && c <= 255.0f)) { *flags |= KVC_FLAG_CODE_OVERFLOW; }
    return (uint32_t)(int)c & 0xffu;
}

// quantise 8 halves held in a uint4 -> 8 code bytes in a uint2; optional smem histogram.
// PS: 0 = the eight values share one unit (p[0]), 1 = value i belongs to unit p[i].  mi2: 512 + min_int (mid_of).
//
// Packed path, for units whose min_int lies in -255..255 (`small_min`; mi2 holds 512 + min_int as fp16 pairs):
// after the fp32 product q0 = x * (1 / scale) everything is done on two values per instruction in fp16, which
// is what the reference's tensors hold anyway.
//  * fp16(q0) equals the reference's fp16(x / scale) except on exact ties between two fp16 subnormals, where
//    both round to the integer 0 (checked over every pair of fp16 values).
//  * qh + 1536 in fp16 is rint(qh) + 1536, exactly, for |qh| <= 512, and 512 + min_int is exact, so their difference t is 1024 + code: the bit pattern
//    0x6400 + code for codes 0 .. 1023, whose low byte is the code; one comparison over all eight tells whether every code is in 0 .. 255.  Beyond 512 the sum is
//    2048 or more and t above 1280, below -512 the sum is below 1024 and t below 768: such values fail the comparison.
//    (With rint(qh), the code and 1024 + code one after the other, 268 MB of keys 183.6 us and of values 114, now 177 and 104.6, a launch's 15 us included.)
// Anything else (a value out of range, not finite, a unit with a large min_int) takes the fp32 path below it,
// which follows the reference's arithmetic to the end.
__device__ __forceinline__ float mid_of(float mi) { return 512.0f + mi; }
// the bit patterns of 1024 + code of two values from their quotients; mid: 512 + min_int
__device__ __forceinline__ uint32_t code_pair(float q0, float q1, const __half2 &mid) {
    const __half2 t = __hsub2_rn(__hadd2_rn(__floats2half2_rn(q0, q1), __float2half2_rn(1536.0f)), mid);
    return *reinterpret_cast<const uint32_t *>(&t);
}
template <int PS>
__device__ __forceinline__ uint2 quant_eight(const uint4 &v, const UnitParam *p, bool small_min, const __half2 *mi2,
                                             int *flags, unsigned int *hist) {
    const __half *h = reinterpret_cast<const __half *>(&v);
    uint2 o;
    if (small_min) {
        const __half2 *h2 = reinterpret_cast<const __half2 *>(&v);
        uint32_t u[4], odd = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float2 xf = __half22float2(h2[k]);
            u[k] = code_pair(__fmul_rn(xf.x, p[2 * k * PS].rcp), __fmul_rn(xf.y, p[(2 * k + 1) * PS].rcp), mi2[k * PS]);
            odd |= u[k] ^ 0x64006400u;
        }
        if ((odd & 0xff00ff00u) == 0) {
            if (hist) {
#pragma unroll
                for (int k = 0; k < 4; k++) { atomicAdd(&hist[u[k] & 0xffu], 1u); atomicAdd(&hist[u[k] >> 16 & 0xffu], 1u); }
            }
            o.x = __byte_perm(u[0], u[1], 0x6420);
            o.y = __byte_perm(u[2], u[3], 0x6420);
            return o;
        }
    }
    uint32_t c[8];
    uint32_t odd = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const UnitParam &u = p[i * PS];
        const float xf = __half2float(h[i]);
        const float q0 = __fmul_rn(xf, u.rcp);
        const float q1 = __fmaf_rn(__fmaf_rn(-q0, u.sf, xf), u.rcp, q0);
        const float qh = __half2float(__float2half_rn(q1));
        const float q = __fsub_rn(__fadd_rn(qh, KVC_RINT_MAGIC), KVC_RINT_MAGIC);
        const float d = __fsub_rn(q, u.mi);
        // d as an integer, read from the mantissa: in range exactly when 0 <= d <= 255
        const uint32_t t = (uint32_t)__float_as_int(__fadd_rn(d, KVC_RINT_MAGIC)) - 0x4B400000u;
        odd |= t;
        c[i] = t & 0xffu;
    }
    if (odd > 255u) {
#pragma unroll
        for (int i = 0; i < 8; i++) c[i] = quant_one(h[i], p[i * PS], flags);
    }
    if (hist) {
#pragma unroll
        for (int i = 0; i < 8; i++) atomicAdd(&hist[c[i]], 1u);
    }
    o.x = c[0] | (c[1] << 8) | (c[2] << 16) | (c[3] << 24);
    o.y = c[4] | (c[5] << 8) | (c[6] << 16) | (c[7] << 24);
    return o;
}
__device__ __forceinline__ bool small_min_int(float mi) { return mi >= -255.0f && mi <= 255.0f; }

// The CTA's bins are private to each warp (sh[warp][256]): fewer lanes meet on a counter.
__device__ __forceinline__ void hist_clear(unsigned int *sh, int tid, int nthr) {
    for (int i = tid; i < (nthr / 32) * 256; i += nthr) sh[i] = 0;
    __syncthreads();
}
__device__ __forceinline__ void hist_flush(const unsigned int *sh, unsigned long long *gh, int tid, int nthr) {
    __syncthreads();
    for (int i = tid; i < 256; i += nthr) {
        unsigned int c = 0;
        for (int w = 0; w < nthr / 32; w++) c += sh[w * 256 + i];
        if (c) atomicAdd(&gh[i], (unsigned long long)c);
    }
}

// extremes of 8 halves: packed fp16 min / max (exact, a NaN operand yields the other one, as fminf does),
// widened once at the end
__device__ __forceinline__ void minmax8(const uint4 &v, float &mn, float &mx) {
    const __half2 *h = reinterpret_cast<const __half2 *>(&v);
    const __half2 lo = __hmin2(__hmin2(h[0], h[1]), __hmin2(h[2], h[3]));
    const __half2 hi = __hmax2(__hmax2(h[0], h[1]), __hmax2(h[2], h[3]));
    mn = fminf(mn, fminf(__low2float(lo), __high2float(lo)));
    mx = fmaxf(mx, fmaxf(__low2float(hi), __high2float(hi)));
}

// ---- ChannelQuant (utils/compute.py:140): one unit per (token block, b, h, channel) -------------
// CTA = one (j, b, h) tile of blk tokens x 128 channels; thread = 8 channels x every 8th token.
// (Measured slower: several tiles per CTA with one flush of the bins; tiles of two or four heads; the tile's
// rows held in registers between the two passes; four rows in flight per thread in either pass.)
// Seven CTAs per SM: 71 registers.  (The tile's place by three 64-bit divisions took 72, and 74 since a code comes from one difference, which leaves room for six:
// 256 columns of 4096 tokens, per head and channel, without and with a histogram 107.4 and 118.6 us, then 112.2 and 125.1, now 98.9 and 109.5; 16 columns of 4096
// 8.5 and 9.5, 9.2 and 10.9, 7.7 and 9.0; one tile 3.6 and 4.1, 3.4 and 3.9, 3.2 and 3.7.)
__global__ void __launch_bounds__(128, 7) quant_channel_kernel(
    const __half *__restrict__ x, long long B, long long H, int blk, float rel,
    uint8_t *__restrict__ codes, void *__restrict__ min_int, int min_bytes, __half *__restrict__ scale,
    unsigned long long *__restrict__ ghist, int *__restrict__ status) {
    __shared__ float smn[8][128], smx[8][128];
    __shared__ unsigned int shist[256];
    const int tid = threadIdx.x, cg = tid & 15, r = tid >> 4;
    const long long row_stride = B * H * 128;
    if (ghist) { for (int i = tid; i < 256; i += 128) shist[i] = 0; }      // a barrier follows before the first count
    int flags = 0;
    const uint32_t tile = blockIdx.x, cols = (uint32_t)(B * H), j = tile / cols;          // (j * B + b) * H + h, below 2^31
    const long long base = ((long long)j * blk * cols + (tile - j * cols)) * 128 + cg * 8;
    __half2 mn2[4], mx2[4];                                 // extremes of the thread's 8 channels, two per register
#pragma unroll
    for (int i = 0; i < 4; i++) { mn2[i] = __float2half2_rn(INFINITY); mx2[i] = __float2half2_rn(-INFINITY); }
    for (int i = r; i < blk; i += 8) {
        uint4 v = *reinterpret_cast<const uint4 *>(x + base + i * row_stride);
        const __half2 *hv = reinterpret_cast<const __half2 *>(&v);
#pragma unroll
        for (int k = 0; k < 4; k++) { mn2[k] = __hmin2(mn2[k], hv[k]); mx2[k] = __hmax2(mx2[k], hv[k]); }
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
        smn[r][cg * 8 + 2 * k] = __low2float(mn2[k]); smn[r][cg * 8 + 2 * k + 1] = __high2float(mn2[k]);
        smx[r][cg * 8 + 2 * k] = __low2float(mx2[k]); smx[r][cg * 8 + 2 * k + 1] = __high2float(mx2[k]);
    }
    __syncthreads();
    {   // thread = channel: fold the 8 partials, derive the unit's parameters once, share them
        float a = smn[0][tid], z = smx[0][tid];
#pragma unroll
        for (int rr = 1; rr < 8; rr++) { a = fminf(a, smn[rr][tid]); z = fmaxf(z, smx[rr][tid]); }
        __half sc;
        const UnitParam q = unit_param(a, z, rel, &sc, &flags);
        const long long u = tile * 128ll + tid;
        scale[u] = sc;
        store_min(min_int, min_bytes, u, q.mi, &flags);
        __syncthreads();                                   // every partial is read before the rows are reused
        smn[0][tid] = q.sf; smn[1][tid] = q.mi; smn[2][tid] = q.rcp;
    }
    __syncthreads();
    UnitParam p[8];
#pragma unroll
    for (int k = 0; k < 8; k++) { p[k].sf = smn[0][cg * 8 + k]; p[k].mi = smn[1][cg * 8 + k]; p[k].rcp = smn[2][cg * 8 + k]; }
    bool small = true;
    __half2 mi2[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        small = small && small_min_int(p[2 * k].mi) && small_min_int(p[2 * k + 1].mi);
        mi2[k] = __floats2half2_rn(mid_of(p[2 * k].mi), mid_of(p[2 * k + 1].mi));
    }
    for (int i = r; i < blk; i += 8) {
        uint4 v = *reinterpret_cast<const uint4 *>(x + base + i * row_stride);
        uint2 o = quant_eight<1>(v, p, small, mi2, &flags, ghist ? shist : nullptr);
        *reinterpret_cast<uint2 *>(codes + base + i * row_stride) = o;
    }
    if (flags) atomicOr(status, flags);
    if (ghist) {
        __syncthreads();
        for (int i = tid; i < 256; i += 128)
            if (shist[i]) atomicAdd(&ghist[i], (unsigned long long)shist[i]);
    }
}

// ---- units that are contiguous runs of `ulen` elements -----------------------------------------
// TokenQuant (all of a token's [B,]H,D values) and VectorQuant (one head's D values).
// GROUP threads share one unit: a warp for short units, the whole CTA (256) for long ones.
template <int GROUP>
__global__ void __launch_bounds__(256) quant_contig_kernel(
    const __half *__restrict__ x, long long n_units, long long ulen, float rel,
    uint8_t *__restrict__ codes, void *__restrict__ min_int, int min_bytes, __half *__restrict__ scale,
    unsigned long long *__restrict__ ghist, int *__restrict__ status) {
    __shared__ float red[2][8];
    __shared__ unsigned int shist[8 * 256];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int UNITS_PER_CTA = 256 / GROUP;
    const long long u = (long long)blockIdx.x * UNITS_PER_CTA + (GROUP == 256 ? 0 : warp);
    const int gl = GROUP == 256 ? tid : lane;          // index inside the group
    if (ghist) hist_clear(shist, tid, 256);
    const bool active = u < n_units;
    const long long chunks = ulen / 8;
    const __half *xu = x + u * ulen;
    float mn = INFINITY, mx = -INFINITY;
    if (active)
        for (long long k = gl; k < chunks; k += GROUP) {
            uint4 v = *reinterpret_cast<const uint4 *>(xu + k * 8);
            minmax8(v, mn, mx);
        }
    mn = -kvc_warp_max(-mn); mx = kvc_warp_max(mx);
    if (GROUP == 256) {
        if (lane == 0) { red[0][warp] = mn; red[1][warp] = mx; }
        __syncthreads();
        mn = red[0][0]; mx = red[1][0];
#pragma unroll
        for (int w = 1; w < 8; w++) { mn = fminf(mn, red[0][w]); mx = fmaxf(mx, red[1][w]); }
    }
    int flags = 0;
    if (active) {
        __half sc;
        UnitParam p = unit_param(mn, mx, rel, &sc, &flags);
        if (gl == 0) { scale[u] = sc; store_min(min_int, min_bytes, u, p.mi, &flags); }
        const bool small = small_min_int(p.mi);
        const __half2 mi2 = __float2half2_rn(mid_of(p.mi));
        for (long long k = gl; k < chunks; k += GROUP) {
            uint4 v = *reinterpret_cast<const uint4 *>(xu + k * 8);
            uint2 o = quant_eight<0>(v, &p, small, &mi2, &flags, ghist ? shist + warp * 256 : nullptr);
            *reinterpret_cast<uint2 *>(codes + u * ulen + k * 8) = o;
        }
    }
    if (flags) atomicOr(status, flags);
    if (ghist) hist_flush(shist, ghist, tid, 256);
}

// Units of CH * WARPS * 256 elements held in registers between the min/max pass and the quantising
// pass (CH 16-byte chunks per thread).  WARPS = 1: a warp per unit, 8 units per 256-thread CTA, nothing
// but shuffles shared.  WARPS > 1: a CTA of WARPS warps per unit, one barrier to join their extremes.
template <int CH, int WARPS>
__global__ void __launch_bounds__(WARPS == 1 ? 256 : WARPS * 32) quant_contig_reg_kernel(
    const __half *__restrict__ x, long long n_units, float rel,
    uint8_t *__restrict__ codes, void *__restrict__ min_int, int min_bytes, __half *__restrict__ scale,
    unsigned long long *__restrict__ ghist, int *__restrict__ status) {
    constexpr int NT = WARPS == 1 ? 256 : WARPS * 32;       // threads per CTA
    constexpr int GT = WARPS * 32;                          // threads per unit
    constexpr long long ULEN = (long long)CH * GT * 8;
    __shared__ unsigned int shist[(NT / 32) * 256];
    __shared__ float red[2][WARPS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gt = WARPS == 1 ? lane : tid;                 // index inside the unit
    if (ghist) hist_clear(shist, tid, NT);
    int flags = 0;
    const long long u_step = WARPS == 1 ? (long long)gridDim.x * 8 : (long long)gridDim.x;
    // every thread of the CTA runs the same number of rounds (the barrier below), units past the end idle
    for (long long u0 = WARPS == 1 ? (long long)blockIdx.x * 8 : (long long)blockIdx.x; u0 < n_units; u0 += u_step) {
    const long long u = WARPS == 1 ? u0 + warp : u0;
    const bool active = u < n_units;
    const __half *xu = x + u * ULEN;
    uint4 v[CH];
    float mn = INFINITY, mx = -INFINITY;
    if (active) {
#pragma unroll
        for (int i = 0; i < CH; i++) v[i] = *reinterpret_cast<const uint4 *>(xu + (long long)(i * GT + gt) * 8);
#pragma unroll
        for (int i = 0; i < CH; i++) minmax8(v[i], mn, mx);
    }
    mn = -kvc_warp_max(-mn); mx = kvc_warp_max(mx);
    if (WARPS > 1) {
        if (lane == 0) { red[0][warp] = mn; red[1][warp] = mx; }
        __syncthreads();
        mn = red[0][0]; mx = red[1][0];
#pragma unroll
        for (int w = 1; w < WARPS; w++) { mn = fminf(mn, red[0][w]); mx = fmaxf(mx, red[1][w]); }
    }
    if (active) {
        __half sc;
        const UnitParam p = unit_param(mn, mx, rel, &sc, &flags);
        if (gt == 0) { scale[u] = sc; store_min(min_int, min_bytes, u, p.mi, &flags); }
        const bool small = small_min_int(p.mi);
        const __half2 mi2 = __float2half2_rn(mid_of(p.mi));
#pragma unroll
        for (int i = 0; i < CH; i++) {
            const uint2 o = quant_eight<0>(v[i], &p, small, &mi2, &flags, ghist ? shist + warp * 256 : nullptr);
            *reinterpret_cast<uint2 *>(codes + u * ULEN + (long long)(i * GT + gt) * 8) = o;
        }
    }
    if (WARPS > 1) __syncthreads();                         // the extremes are read before the next unit's
    }
    if (flags) atomicOr(status, flags);
    if (ghist) hist_flush(shist, ghist, tid, NT);
}

// ---- BlockQuant: one unit per token block (x sequence), far larger than a CTA ------------------
// Three launches: per-row min/max folded into the unit with atomics on order-preserving keys,
// a per-unit finalise, and the elementwise pass.  A row is one (token, b): H*D contiguous values.
// The same three serve the two-call form (kvc_quant_minmax / kvc_quantize_ranged) for every unit made of
// whole rows: `blk` is then the unit's token divisor (the block for BlockQuant, 1 for TokenQuant).
__device__ __forceinline__ unsigned int half_key(float f) {      // monotone in the value
    unsigned int h = __half_as_ushort(__float2half_rn(f));
    return (h & 0x8000u) ? (~h & 0xffffu) : (h | 0x8000u);
}
__device__ __forceinline__ float key_half(unsigned int k) {
    unsigned int h = (k & 0x8000u) ? (k & 0x7fffu) : (~k & 0xffffu);
    return __half2float(__ushort_as_half((unsigned short)h));
}

__global__ void __launch_bounds__(256) quant_block_minmax_kernel(
    const __half *__restrict__ x, long long B, long long row_len, int blk, int batch_shared,
    unsigned int *__restrict__ ws) {
    __shared__ float red[2][8];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long row = blockIdx.x, t = row / B, b = row % B;
    const long long u = batch_shared ? t / blk : (t / blk) * B + b;
    const __half *xr = x + row * row_len;
    float mn = INFINITY, mx = -INFINITY;
    for (long long k = tid; k < row_len / 8; k += 256) {
        uint4 v = *reinterpret_cast<const uint4 *>(xr + k * 8);
        minmax8(v, mn, mx);
    }
    mn = -kvc_warp_max(-mn); mx = kvc_warp_max(mx);
    if (lane == 0) { red[0][warp] = mn; red[1][warp] = mx; }
    __syncthreads();
    if (tid == 0) {
#pragma unroll
        for (int w = 1; w < 8; w++) { mn = fminf(mn, red[0][w]); mx = fmaxf(mx, red[1][w]); }
        atomicMax(&ws[2 * u], 0xffffu - half_key(mn));     // max of the inverted key == min of the value
        atomicMax(&ws[2 * u + 1], half_key(mx));
    }
}

// keys -> the units' extremes as fp16 (what ranks exchange when a unit spans the heads of several of them)
__global__ void quant_minmax_export_kernel(const unsigned int *__restrict__ ws, long long n_units,
                                           __half *__restrict__ mn_out, __half *__restrict__ mx_out) {
    long long u = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= n_units) return;
    mn_out[u] = __float2half_rn(key_half(0xffffu - ws[2 * u]));
    mx_out[u] = __float2half_rn(key_half(ws[2 * u + 1]));
}

// mn_in / mx_in (optional): the units' extremes given by the caller instead of the keys in ws
__global__ void quant_block_finalize_kernel(unsigned int *__restrict__ ws, long long n_units, float rel,
                                            void *__restrict__ min_int, int min_bytes,
                                            __half *__restrict__ scale, int *__restrict__ status,
                                            const __half *__restrict__ mn_in, const __half *__restrict__ mx_in) {
    long long u = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= n_units) return;
    float mn, mx;
    if (mn_in) { mn = __half2float(mn_in[u]); mx = __half2float(mx_in[u]); }
    else { mn = key_half(0xffffu - ws[2 * u]); mx = key_half(ws[2 * u + 1]); }
    int flags = 0;
    __half sc;
    UnitParam p = unit_param(mn, mx, rel, &sc, &flags);
    scale[u] = sc;
    store_min(min_int, min_bytes, u, p.mi, &flags);
    // leave the unit parameters where the elementwise pass reads them
    ws[2 * u] = __float_as_uint(p.sf);
    ws[2 * u + 1] = __float_as_uint(p.mi);
    if (flags) atomicOr(status, flags);
}

__global__ void __launch_bounds__(256) quant_block_apply_kernel(
    const __half *__restrict__ x, long long B, long long row_len, int blk, int batch_shared,
    const unsigned int *__restrict__ ws, uint8_t *__restrict__ codes,
    unsigned long long *__restrict__ ghist, int *__restrict__ status) {
    __shared__ unsigned int shist[8 * 256];
    const int tid = threadIdx.x;
    const long long row = blockIdx.x, t = row / B, b = row % B;
    const long long u = batch_shared ? t / blk : (t / blk) * B + b;
    if (ghist) hist_clear(shist, tid, 256);
    UnitParam p;
    p.sf = __uint_as_float(ws[2 * u]); p.mi = __uint_as_float(ws[2 * u + 1]);
    p.rcp = (p.sf == 0.0f || p.sf != p.sf) ? 0.0f : __frcp_rn(p.sf);
    int flags = 0;
    const bool small = small_min_int(p.mi);
    const __half2 mi2 = __float2half2_rn(mid_of(p.mi));
    for (long long k = tid; k < row_len / 8; k += 256) {
        uint4 v = *reinterpret_cast<const uint4 *>(x + row * row_len + k * 8);
        uint2 o = quant_eight<0>(v, &p, small, &mi2, &flags, ghist ? shist + (tid >> 5) * 256 : nullptr);
        *reinterpret_cast<uint2 *>(codes + row * row_len + k * 8) = o;
    }
    if (flags) atomicOr(status, flags);
    if (ghist) hist_flush(shist, ghist, tid, 256);
}

// Eight channels of the lower half (xa) and their partners of the upper half (xb), rotated with torch's roundings: t * cos +
// rotate_half(t) * sin, each op rounded to fp16.  (Torch computes an op in fp32 and rounds: the same fp16 value as one
// rounding, for a product because it is exact in fp32, for a sum because fp32 has more than twice fp16's digits; the _rn forms
// are never contracted into a fused multiply-add.  Through fp32 this took three times the instructions.)
__device__ __forceinline__ void rope8(const uint4 &xa, const uint4 &xb, const uint4 &ca, const uint4 &cb, const uint4 &sa, const uint4 &sb,
                                      uint4 &oa, uint4 &ob) {
    const __half2 *x1 = reinterpret_cast<const __half2 *>(&xa), *x2 = reinterpret_cast<const __half2 *>(&xb);
    const __half2 *c1 = reinterpret_cast<const __half2 *>(&ca), *c2 = reinterpret_cast<const __half2 *>(&cb);
    const __half2 *s1 = reinterpret_cast<const __half2 *>(&sa), *s2 = reinterpret_cast<const __half2 *>(&sb);
    uint4 a, b;
    __half2 *o1 = reinterpret_cast<__half2 *>(&a), *o2 = reinterpret_cast<__half2 *>(&b);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        // rotate_half: the lower half meets -x2, the upper half x1
        o1[k] = __hadd2_rn(__hmul2_rn(x1[k], c1[k]), __hmul2_rn(__hneg2(x2[k]), s1[k]));
        o2[k] = __hadd2_rn(__hmul2_rn(x2[k], c2[k]), __hmul2_rn(x1[k], s2[k]));
    }
    oa = a; ob = b;
}

// ---- a prompt, quantised where its projections left it --------------------------------------------
// x [B, H, Tx, 128] (heads first), the first T tokens of it -> codes [T, B, H, 128] (tokens first), keys rotated on the way.
// Bound by memory: 2 bytes read and 1 written per value, where a rotated and transposed copy of the tensor took 4 more before
// the quantiser read it (K per channel: twice).

// The CTA's histogram: codes below 32 are counted two at a time, n[first + 39 * second], others one by one behind these
// counters, n[PAIR_BINS + code] (three instructions per code one by one, a good half of that for a pair; fewer lanes meet on a counter).  39: the codes of a
// unit are a bell curve, and with rows of 32 counters every pair of one first code lies in one bank (268 MB of keys 189 us, with 39 183.6; of values 116.3 and 114).
constexpr int PAIR_ROW = 39, PAIR_BINS = 31 + 31 * PAIR_ROW + 1;
struct PairBins { unsigned int n[PAIR_BINS + 256]; };
__device__ __forceinline__ void bins_clear(PairBins &b, int tid, int nthr) {
    for (int i = tid; i < PAIR_BINS + 256; i += nthr) b.n[i] = 0;
    __syncthreads();
}
__device__ __forceinline__ void bins_add(PairBins &b, const uint32_t (&u)[4]) {     // two codes per word, in the low bytes of its halves
    if (((u[0] | u[1] | u[2] | u[3]) & 0x00e000e0u) == 0) {
#pragma unroll
        for (int k = 0; k < 4; k++) atomicAdd(reinterpret_cast<unsigned int *>(reinterpret_cast<char *>(b.n) + __dp4a(u[k], (uint32_t)(4 * PAIR_ROW << 16 | 4), 0u)), 1u);
    } else {
#pragma unroll
        for (int k = 0; k < 4; k++) { atomicAdd(&b.n[PAIR_BINS + (u[k] & 0xffu)], 1u); atomicAdd(&b.n[PAIR_BINS + (u[k] >> 16 & 0xffu)], 1u); }
    }
}
__device__ __forceinline__ void bins_flush(const PairBins &b, unsigned long long *gh, int tid) {      // by the first 256 threads
    __syncthreads();
    if (tid >= 256) return;
    unsigned int c = 0;
    const int s = tid >> 3, part = tid & 7;                 // eight threads fold a symbol's row and column
#pragma unroll
    for (int k = 0; k < 4; k++) c += b.n[s + PAIR_ROW * (part * 4 + k)] + b.n[PAIR_ROW * s + part * 4 + k];
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if (part == 0 && c) atomicAdd(&gh[s], (unsigned long long)c);
    if (b.n[PAIR_BINS + tid]) atomicAdd(&gh[tid], (unsigned long long)b.n[PAIR_BINS + tid]);
}

// the packed path of quant_eight with what it needs in registers; param(i): value i's unit, for anything else
template <class P>
__device__ __forceinline__ uint2 quant_eight_at(const uint4 &v, const float (&rcp)[8], const __half2 (&mi2)[4], bool small_min, P param,
                                                int *flags, PairBins *bins) {
    const __half2 *h2 = reinterpret_cast<const __half2 *>(&v);
    uint32_t u[4], odd = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float2 xf = __half22float2(h2[k]);
        u[k] = code_pair(__fmul_rn(xf.x, rcp[2 * k]), __fmul_rn(xf.y, rcp[2 * k + 1]), mi2[k]);
        odd |= u[k] ^ 0x64006400u;
    }
    if (!small_min || (odd & 0xff00ff00u) != 0) {
        const __half *h = reinterpret_cast<const __half *>(&v);
#pragma unroll
        for (int k = 0; k < 4; k++) u[k] = quant_one(h[2 * k], param(2 * k), flags) | (quant_one(h[2 * k + 1], param(2 * k + 1), flags) << 16);
    }
    if (bins) bins_add(*bins, u);
    return make_uint2(__byte_perm(u[0], u[1], 0x6420), __byte_perm(u[2], u[3], 0x6420));
}

// ChannelQuant.  CTA = THREADS / 8 * ROWS tokens (one block) of `heads` heads, one after the other; thread = 8 channels of either
// half of ROWS rows, whose cos and sin it keeps; the next head's rows are fetched while this one's are at work.
// (Issue bounds it, with 128 registers two CTAs per SM: 1 GiB of keys 0.62 ms, values 0.34 ms by
// quant_heads_token_kernel; copies and the quantisers of rows took 1.17 and 0.79.  80 registers, three CTAs: 5 % slower.)
template <int ROWS, int THREADS, bool ROPE>
__global__ void __launch_bounds__(THREADS, 512 / THREADS) quant_heads_channel_kernel(
    const __half *__restrict__ x, const __half *__restrict__ cs, const __half *__restrict__ sn, long long cs_bstride,
    uint32_t B, uint32_t H, uint32_t heads, long long Tx, float rel, uint8_t *__restrict__ codes, void *__restrict__ min_int,
    int min_bytes, __half *__restrict__ scale, unsigned long long *__restrict__ ghist, int *__restrict__ status) {
    constexpr int WARPS = THREADS / 32, RT = THREADS / 8;   // RT: rows side by side
    __shared__ __align__(16) __half smn[WARPS][128], smx[WARPS][128];
    __shared__ __align__(16) float psf[128], pmi[128], prcp[128];
    __shared__ __align__(16) __half phm[128];               // mid_of(min_int) of the units of psmall
    __shared__ unsigned int psmall[4];                      // a bit per channel: small_min_int
    __shared__ PairBins bins;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, cg = tid & 7, r = tid >> 3;
    const uint32_t groups = (H + heads - 1) / heads, b = blockIdx.x / groups, h0 = (blockIdx.x % groups) * heads, h1 = min(H, h0 + heads);
    const long long j = blockIdx.y, tok0 = j * (RT * ROWS) + r;
    if (ghist) bins_clear(bins, tid, THREADS);
    uint4 ca[ROWS], cb[ROWS], sa[ROWS], sb[ROWS];
    if (ROPE) {
#pragma unroll
        for (int k = 0; k < ROWS; k++) {
            const __half *c = cs + b * cs_bstride + (tok0 + RT * k) * 128 + cg * 8, *s = sn + b * cs_bstride + (tok0 + RT * k) * 128 + cg * 8;
            ca[k] = *reinterpret_cast<const uint4 *>(c); cb[k] = *reinterpret_cast<const uint4 *>(c + 64);
            sa[k] = *reinterpret_cast<const uint4 *>(s); sb[k] = *reinterpret_cast<const uint4 *>(s + 64);
        }
    }
    uint4 na[ROWS], nb[ROWS];
    auto fetch = [&](uint32_t h) {
        const __half *xr = x + (((long long)b * H + h) * Tx + tok0) * 128 + cg * 8;
#pragma unroll
        for (int k = 0; k < ROWS; k++) { na[k] = *reinterpret_cast<const uint4 *>(xr + k * (RT * 128)); nb[k] = *reinterpret_cast<const uint4 *>(xr + k * (RT * 128) + 64); }
    };
    fetch(h0);
    uint8_t *const out0 = codes + ((tok0 * B + b) * H) * 128 + cg * 8;
    const size_t out_row = (size_t)RT * B * H * 128;
    int flags = 0;
    for (uint32_t h = h0; h < h1; h++) {
        uint4 va[ROWS], vb[ROWS];
#pragma unroll
        for (int k = 0; k < ROWS; k++) {
            if (ROPE) rope8(na[k], nb[k], ca[k], cb[k], sa[k], sb[k], va[k], vb[k]);
            else { va[k] = na[k]; vb[k] = nb[k]; }
        }
        if (h + 1 < h1) fetch(h + 1);
        // extremes of the thread's 16 channels, then of the warp's four row groups: at each step a lane gives half of its
        // channels away and keeps the other half, so that each ends with four channels' extremes
        __half2 mn[8], mx[8];                               // 0..3: the lower half's channel pairs, 4..7: the upper half's
#pragma unroll
        for (int i = 0; i < 4; i++) {
            mn[i] = mx[i] = reinterpret_cast<const __half2 *>(&va[0])[i]; mn[4 + i] = mx[4 + i] = reinterpret_cast<const __half2 *>(&vb[0])[i];
#pragma unroll
            for (int k = 1; k < ROWS; k++) {
                const __half2 p = reinterpret_cast<const __half2 *>(&va[k])[i], q = reinterpret_cast<const __half2 *>(&vb[k])[i];
                mn[i] = __hmin2(mn[i], p); mx[i] = __hmax2(mx[i], p); mn[4 + i] = __hmin2(mn[4 + i], q); mx[4 + i] = __hmax2(mx[4 + i], q);
            }
        }
        const bool up = (lane & 16) != 0, odd = (lane & 8) != 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const __half2 gn = __shfl_xor_sync(0xffffffffu, up ? mn[i] : mn[4 + i], 16), gx = __shfl_xor_sync(0xffffffffu, up ? mx[i] : mx[4 + i], 16);
            mn[i] = __hmin2(up ? mn[4 + i] : mn[i], gn); mx[i] = __hmax2(up ? mx[4 + i] : mx[i], gx);
        }
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const __half2 gn = __shfl_xor_sync(0xffffffffu, odd ? mn[i] : mn[2 + i], 8), gx = __shfl_xor_sync(0xffffffffu, odd ? mx[i] : mx[2 + i], 8);
            mn[i] = __hmin2(odd ? mn[2 + i] : mn[i], gn); mx[i] = __hmax2(odd ? mx[2 + i] : mx[i], gx);
        }
        const int at = (up ? 64 : 0) + cg * 8 + (odd ? 4 : 0);
        *reinterpret_cast<__half2 *>(&smn[warp][at]) = mn[0]; *reinterpret_cast<__half2 *>(&smn[warp][at + 2]) = mn[1];
        *reinterpret_cast<__half2 *>(&smx[warp][at]) = mx[0]; *reinterpret_cast<__half2 *>(&smx[warp][at + 2]) = mx[1];
        __syncthreads();                                    // (also: the head before is done with its units' parameters)
        if (tid < 128) {                                    // thread = channel
            const int at2 = tid & ~1;
            // (from the infinities: a channel of nothing but NaN has the extremes +inf and -inf, as in quant_channel_kernel)
            __half2 a = __float2half2_rn(INFINITY), z = __float2half2_rn(-INFINITY);
#pragma unroll
            for (int w = 0; w < WARPS; w++) { a = __hmin2(a, *reinterpret_cast<const __half2 *>(&smn[w][at2])); z = __hmax2(z, *reinterpret_cast<const __half2 *>(&smx[w][at2])); }
            __half sc;
            const UnitParam q = unit_param(tid & 1 ? __high2float(a) : __low2float(a), tid & 1 ? __high2float(z) : __low2float(z), rel, &sc, &flags);
            const long long u = ((j * B + b) * H + h) * 128 + tid;
            scale[u] = sc;
            store_min(min_int, min_bytes, u, q.mi, &flags);
            psf[tid] = q.sf; pmi[tid] = q.mi; prcp[tid] = q.rcp; phm[tid] = __float2half_rn(mid_of(q.mi));
            const unsigned int small = __ballot_sync(0xffffffffu, small_min_int(q.mi));
            if (lane == 0) psmall[warp] = small;
        }
        __syncthreads();
#pragma unroll
        for (int half = 0; half < 2; half++) {
            const int c0 = half * 64 + cg * 8;
            float rcp[8];
            __half2 mi2[4];
            const bool small = (psmall[c0 >> 5] >> (c0 & 31) & 0xffu) == 0xffu;
#pragma unroll
            for (int i = 0; i < 8; i += 4) *reinterpret_cast<float4 *>(&rcp[i]) = *reinterpret_cast<const float4 *>(&prcp[c0 + i]);
            *reinterpret_cast<uint4 *>(mi2) = *reinterpret_cast<const uint4 *>(&phm[c0]);
            auto param = [&](int i) { UnitParam p; p.sf = psf[c0 + i]; p.mi = pmi[c0 + i]; p.rcp = prcp[c0 + i]; return p; };
#pragma unroll
            for (int k = 0; k < ROWS; k++) {
                const uint2 o = quant_eight_at(half ? vb[k] : va[k], rcp, mi2, small, param, &flags, ghist ? &bins : nullptr);
                *reinterpret_cast<uint2 *>(out0 + k * out_row + (size_t)h * 128 + half * 64) = o;
            }
        }
    }
    if (flags) atomicOr(status, flags);
    if (ghist) bins_flush(bins, ghist, tid);
}

// TokenQuant (a unit: one token of one sequence, all heads) and VectorQuant (one head of it).  CTA = four tokens of one sequence
// at a time, all heads in registers (NH x 4 at most); thread = 8 channels of one token in every fourth head.
template <int NH, bool VECTOR>
__global__ void __launch_bounds__(256) quant_heads_token_kernel(
    const __half *__restrict__ x, uint32_t B, uint32_t H, long long Tx, long long T, float rel, uint8_t *__restrict__ codes,
    void *__restrict__ min_int, int min_bytes, __half *__restrict__ scale, unsigned long long *__restrict__ ghist,
    int *__restrict__ status) {
    __shared__ float red[2][4][4];                          // extremes by head group and token
    __shared__ PairBins bins;
    const int tid = threadIdx.x, c0 = (tid & 15) * 8, tk = (tid >> 4) & 3, hg = tid >> 6;
    if (ghist) bins_clear(bins, tid, 256);
    int flags = 0;
    const long long n4 = (T + 3) / 4, n_groups = n4 * B;
    for (long long grp = blockIdx.x; grp < n_groups; grp += gridDim.x) {
        const uint32_t b = (uint32_t)(grp / n4);            // neighbouring CTAs: neighbouring tokens of a sequence
        const long long tok = (grp - b * n4) * 4 + tk;
        const bool live = tok < T;
        uint4 v[NH];
        const __half *xr = x + ((long long)b * H * Tx + tok) * 128 + c0;
#pragma unroll
        for (int i = 0; i < NH; i++) {
            const uint32_t h = i * 4 + hg;
            v[i] = make_uint4(0u, 0u, 0u, 0u);
            if (live && h < H) v[i] = *reinterpret_cast<const uint4 *>(xr + h * Tx * 128);
        }
        float mn = INFINITY, mx = -INFINITY;
        UnitParam p = {0.f, 0.f, 0.f};
        if (!VECTOR) {
#pragma unroll
            for (int i = 0; i < NH; i++) if ((uint32_t)(i * 4 + hg) < H) minmax8(v[i], mn, mx);
#pragma unroll
            for (int o = 1; o < 16; o <<= 1) { mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o)); mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o)); }
            __syncthreads();                                // the group before is done with its extremes
            if (c0 == 0) { red[0][hg][tk] = mn; red[1][hg][tk] = mx; }
            __syncthreads();
            mn = fminf(fminf(red[0][0][tk], red[0][1][tk]), fminf(red[0][2][tk], red[0][3][tk]));
            mx = fmaxf(fmaxf(red[1][0][tk], red[1][1][tk]), fmaxf(red[1][2][tk], red[1][3][tk]));
            if (live) {
                __half sc;
                p = unit_param(mn, mx, rel, &sc, &flags);
                if (c0 == 0 && hg == 0) { scale[tok * B + b] = sc; store_min(min_int, min_bytes, tok * B + b, p.mi, &flags); }
            }
        }
#pragma unroll
        for (int i = 0; i < NH; i++) {
            const uint32_t h = i * 4 + hg;
            if (VECTOR) {
                mn = INFINITY; mx = -INFINITY;
                minmax8(v[i], mn, mx);
#pragma unroll
                for (int o = 1; o < 16; o <<= 1) { mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o)); mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o)); }
            }
            if (!live || h >= H) continue;
            const long long u = (tok * B + b) * H + h;      // also the row of the codes
            if (VECTOR) {
                __half sc;
                p = unit_param(mn, mx, rel, &sc, &flags);
                if (c0 == 0) { scale[u] = sc; store_min(min_int, min_bytes, u, p.mi, &flags); }
            }
            const __half2 m2 = __float2half2_rn(mid_of(p.mi));
            const float rcp[8] = {p.rcp, p.rcp, p.rcp, p.rcp, p.rcp, p.rcp, p.rcp, p.rcp};
            const __half2 mi2[4] = {m2, m2, m2, m2};
            *reinterpret_cast<uint2 *>(codes + u * 128 + c0) = quant_eight_at(v[i], rcp, mi2, small_min_int(p.mi), [&](int) { return p; }, &flags, ghist ? &bins : nullptr);
        }
    }
    if (flags) atomicOr(status, flags);
    if (ghist) bins_flush(bins, ghist, tid);
}

// ---- dequantise: fp16((code + min_int) * scale), models/cache/kvcomp_encode.py:146 -------------
// Bound by memory (1 byte in, 2 out).  A thread takes GROUPS groups of 8 channels, all their loads in flight together;
// wide_units: units side by side over the channels, 8 of them fetched with one load per array.  Two groups where the units
// do not depend on the channel and there are enough of them to fill the device, else one: 64 x 128 values 2.1 us (two
// groups 2.3, four 2.9), 33.6 M values 24.0 us (20.3, 20.4); per-channel units, more registers each, 2.3 us (2.7, 3.8) and 30.6
// (33.3, 34.3).  With 64-bit divisions and a load per unit: 2.6 and 42.9, per channel 2.7 and 46.5 us.
template <int GROUPS>
__global__ void __launch_bounds__(256) dequant_kernel(const uint8_t *__restrict__ codes, kvc_qmeta_dev m,
                                                      long long rows, uint32_t B, uint32_t H, uint32_t D, int wide_units,
                                                      __half *__restrict__ out) {
    const uint32_t per_row = D / 8;
    const long long n = rows * per_row, i0 = (long long)blockIdx.x * (256 * GROUPS) + threadIdx.x;
    uint2 cv[GROUPS];
#pragma unroll
    for (int g = 0; g < GROUPS; g++) {
        const long long i = i0 + g * 256;
        if (i < n) cv[g] = *reinterpret_cast<const uint2 *>(codes + i * 8);
    }
#pragma unroll
    for (int g = 0; g < GROUPS; g++) {
        const long long i = i0 + g * 256;
        if (i >= n) return;
        uint32_t c0, h, b;
        long long t;
        if (n < (1ll << 32)) {                               // the same for the whole grid
            uint32_t r = (uint32_t)i / per_row;
            c0 = ((uint32_t)i - r * per_row) * 8;
            h = r % H; r /= H; b = r % B; t = r / B;
        } else {
            long long r = i / per_row;
            c0 = (uint32_t)(i - r * per_row) * 8;
            h = (uint32_t)(r % H); r /= H; b = (uint32_t)(r % B); t = r / B;
        }
        uint4 o;
        if (m.sc == 0) {
            float mi; __half2 sc;
            kvc_row_unit(m, t, b, h, mi, sc);
            o = kvc_dequant8(cv[g].x, cv[g].y, mi, sc);
        } else {
            const long long u = kvc_tok_unit(t, m.tok_div) * m.sj + b * m.sb + h * m.sh + (long long)c0 * m.sc;
            float mi[8];
            __half2 sc[4];
            if (wide_units) {
                const uint4 sv = *reinterpret_cast<const uint4 *>(m.scale + u);
                const __half2 *s2 = reinterpret_cast<const __half2 *>(&sv);
#pragma unroll
                for (int k = 0; k < 4; k++) sc[k] = s2[k];
                if (m.min_bytes == 1) {
                    const uint2 mv = *reinterpret_cast<const uint2 *>(reinterpret_cast<const int8_t *>(m.min_int) + u);
                    const int8_t *mb = reinterpret_cast<const int8_t *>(&mv);
#pragma unroll
                    for (int k = 0; k < 8; k++) mi[k] = (float)mb[k] - 8388608.0f;
                } else {
                    const uint4 mv = *reinterpret_cast<const uint4 *>(reinterpret_cast<const int16_t *>(m.min_int) + u);
                    const int16_t *mh = reinterpret_cast<const int16_t *>(&mv);
#pragma unroll
                    for (int k = 0; k < 8; k++) mi[k] = (float)mh[k] - 8388608.0f;
                }
            } else {
                __half s1[8];
#pragma unroll
                for (int k = 0; k < 8; k++) { mi[k] = (float)kvc_load_min(m, u + k * m.sc) - 8388608.0f; s1[k] = m.scale[u + k * m.sc]; }
#pragma unroll
                for (int k = 0; k < 4; k++) sc[k] = __halves2half2(s1[2 * k], s1[2 * k + 1]);
            }
            o = kvc_dequant8(cv[g].x, cv[g].y, mi, sc);
        }
        *reinterpret_cast<uint4 *>(out + i * 8) = o;
    }
}

// ---- dense q.k over uncompressed K (kernels.cu:1192-1219), fp32 accumulation --------------------
// One warp per (token, head) row of 128 fp16 values; lane = 4 channels.
__global__ void __launch_bounds__(256) k_matvec_kernel(const __half *__restrict__ k, const __half *__restrict__ q,
                                                       __half *__restrict__ out, long long rows, long long H) {
    const int lane = threadIdx.x & 31;
    long long row = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= rows) return;
    uint2 kv = *reinterpret_cast<const uint2 *>(k + row * 128 + lane * 4);
    uint2 qv = *reinterpret_cast<const uint2 *>(q + (row % H) * 128 + lane * 4);
    const __half2 *k2 = reinterpret_cast<const __half2 *>(&kv), *q2 = reinterpret_cast<const __half2 *>(&qv);
    float acc = 0.f;
#pragma unroll
    for (int i = 0; i < 2; i++) {
        float2 a = __half22float2(k2[i]), c = __half22float2(q2[i]);
        acc = fmaf(a.x, c.x, acc); acc = fmaf(a.y, c.y, acc);
    }
    acc = kvc_warp_sum(acc);
    if (lane == 0) out[row] = __float2half_rn(acc);
}

}  // namespace

extern "C" int kvc_qmeta_make(int mode, int batch_shared, int64_t T, int64_t B, int64_t H, int64_t D,
                              int64_t block, kvc_qmeta *q, int64_t *n_units) {
    KVC_REQUIRE(q != nullptr, "kvc_qmeta_make: q is null");
    KVC_REQUIRE(T >= 0 && B > 0 && H > 0 && D > 0, "kvc_qmeta_make: bad shape");
    const int64_t nb = batch_shared ? 1 : B;
    int64_t n = 0;
    q->sj = q->sb = q->sh = q->sc = 0;
    switch (mode) {
    case KVC_MODE_BLOCK:
        KVC_REQUIRE(block > 0 && T % block == 0, "kvc_qmeta_make: T=%lld is not a multiple of block=%lld", (long long)T, (long long)block);
        q->tok_div = (int32_t)block; q->sj = nb; q->sb = batch_shared ? 0 : 1; n = (T / block) * nb; break;
    case KVC_MODE_CHANNEL:
        KVC_REQUIRE(block > 0 && T % block == 0, "kvc_qmeta_make: T=%lld is not a multiple of block=%lld", (long long)T, (long long)block);
        q->tok_div = (int32_t)block; q->sj = B * H * D; q->sb = H * D; q->sh = D; q->sc = 1; n = (T / block) * B * H * D; break;
    case KVC_MODE_TOKEN:
        q->tok_div = 1; q->sj = nb; q->sb = batch_shared ? 0 : 1; n = T * nb; break;
    case KVC_MODE_VECTOR:
        q->tok_div = 1; q->sj = B * H; q->sb = H; q->sh = 1; n = T * B * H; break;
    default:
        KVC_REQUIRE(false, "kvc_qmeta_make: unknown mode %d", mode);
    }
    if (n_units) *n_units = n;
    return KVC_OK;
}

extern "C" int64_t kvc_quantize_workspace(int mode, int batch_shared, int64_t T, int64_t B, int64_t block) {
    if (mode != KVC_MODE_BLOCK || block <= 0) return 0;
    return (T / block) * (batch_shared ? 1 : B) * 8;
}

extern "C" int kvc_quantize(const void *x, int64_t T, int64_t B, int64_t H, int64_t D,
                            int mode, int batch_shared, int64_t block, float rel,
                            uint8_t *codes, void *min_int, int min_bytes, void *scale,
                            unsigned long long *hist, void *workspace, int64_t workspace_bytes,
                            int32_t *status, kvc_stream_t stream) {
    KVC_REQUIRE(x && codes && min_int && scale && status, "kvc_quantize: null pointer");
    KVC_REQUIRE(T >= 0 && B > 0 && H > 0 && D > 0 && D % 8 == 0, "kvc_quantize: bad shape T=%lld B=%lld H=%lld D=%lld", (long long)T, (long long)B, (long long)H, (long long)D);
    KVC_REQUIRE(min_bytes == 1 || min_bytes == 2, "kvc_quantize: min_bytes must be 1 or 2");
    KVC_REQUIRE((reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(codes) & 7) == 0,
                "kvc_quantize: x must be 16-byte and codes 8-byte aligned");
    if (T == 0) return KVC_OK;
    cudaStream_t s = kvc_cu(stream);
    const __half *xh = reinterpret_cast<const __half *>(x);
    __half *sc = reinterpret_cast<__half *>(scale);
    switch (mode) {
    case KVC_MODE_CHANNEL: {
        KVC_REQUIRE(D == 128, "kvc_quantize: ChannelQuant needs head_dim 128");
        KVC_REQUIRE(block > 0 && T % block == 0, "kvc_quantize: T=%lld is not a multiple of block=%lld", (long long)T, (long long)block);
        long long tiles = (T / block) * B * H;
        KVC_REQUIRE(tiles < (1ll << 31), "kvc_quantize: too many tiles");
        quant_channel_kernel<<<(unsigned)tiles, 128, 0, s>>>(xh, B, H, (int)block, rel, codes, min_int, min_bytes, sc, hist, status);
        break;
    }
    case KVC_MODE_TOKEN:
    case KVC_MODE_VECTOR: {
        long long ulen = mode == KVC_MODE_VECTOR ? D : (batch_shared ? B * H * D : H * D);
        long long n_units = T * B * H * D / ulen;
#define KVC_QR(CH_, W_) quant_contig_reg_kernel<CH_, W_><<<(unsigned)std::min<long long>((W_) == 1 ? (n_units + 7) / 8 : n_units, (long long)kvc_sm_count() * (2048 / ((W_) == 1 ? 256 : (W_) * 32))), (W_) == 1 ? 256 : (W_) * 32, 0, s>>>( \
        xh, n_units, rel, codes, min_int, min_bytes, sc, hist, status)
        if (n_units < (1ll << 31) && (ulen == 256 || ulen == 512 || ulen == 1024 || ulen == 2048 || ulen == 4096 || ulen == 8192)) {
            switch (ulen) {
            case 256: KVC_QR(1, 1); break;
            case 512: KVC_QR(2, 1); break;
            case 1024: KVC_QR(4, 1); break;
            case 2048: KVC_QR(4, 2); break;
            case 4096: KVC_QR(4, 4); break;
            default: KVC_QR(4, 8); break;
            }
        } else
#undef KVC_QR
        if (ulen >= 2048) {
            KVC_REQUIRE(n_units < (1ll << 31), "kvc_quantize: too many units");
            quant_contig_kernel<256><<<(unsigned)n_units, 256, 0, s>>>(xh, n_units, ulen, rel, codes, min_int, min_bytes, sc, hist, status);
        } else {
            long long ctas = (n_units + 7) / 8;
            KVC_REQUIRE(ctas < (1ll << 31), "kvc_quantize: too many units");
            quant_contig_kernel<32><<<(unsigned)ctas, 256, 0, s>>>(xh, n_units, ulen, rel, codes, min_int, min_bytes, sc, hist, status);
        }
        break;
    }
    case KVC_MODE_BLOCK: {
        KVC_REQUIRE(block > 0 && T % block == 0, "kvc_quantize: T=%lld is not a multiple of block=%lld", (long long)T, (long long)block);
        long long n_units = (T / block) * (batch_shared ? 1 : B);
        KVC_REQUIRE(workspace && workspace_bytes >= n_units * 8, "kvc_quantize: BlockQuant needs %lld bytes of workspace", n_units * 8);
        KVC_REQUIRE(T * B < (1ll << 31), "kvc_quantize: too many rows");
        unsigned int *ws = reinterpret_cast<unsigned int *>(workspace);
        KVC_CUDA_OK(cudaMemsetAsync(ws, 0, n_units * 8, s));
        quant_block_minmax_kernel<<<(unsigned)(T * B), 256, 0, s>>>(xh, B, H * D, (int)block, batch_shared, ws);
        quant_block_finalize_kernel<<<(unsigned)((n_units + 127) / 128), 128, 0, s>>>(ws, n_units, rel, min_int, min_bytes, sc, status, nullptr, nullptr);
        quant_block_apply_kernel<<<(unsigned)(T * B), 256, 0, s>>>(xh, B, H * D, (int)block, batch_shared, ws, codes, hist, status);
        break;
    }
    default:
        KVC_REQUIRE(false, "kvc_quantize: unknown mode %d", mode);
    }
    KVC_LAUNCH_OK();
    return KVC_OK;
}

// The same for units side by side over the channels that cover TOKENS tokens or more: a thread's eight channels have the same units in all of them, so a
// thread loads them once and has TOKENS loads of codes in flight.  (512 rows of 32 x 32 heads, 67 M values: 56 us where a thread takes the channels of one
// token, now 33.)
namespace {
template <int TOKENS>
__global__ void __launch_bounds__(256) dequant_channel_kernel(const uint8_t *__restrict__ codes, kvc_qmeta_dev m, uint32_t H, uint32_t per_head, uint32_t per_token,
                                                              __half *__restrict__ out) {
    const uint32_t c = blockIdx.x * 256 + threadIdx.x;      // eight channels of a token's row
    if (c >= per_token) return;
    const long long t0 = (long long)blockIdx.y * TOKENS;
    const uint32_t c0 = (c % per_head) * 8, col = c / per_head, h = col % H, b = col / H;
    uint2 cv[TOKENS];
#pragma unroll
    for (int k = 0; k < TOKENS; k++) cv[k] = *reinterpret_cast<const uint2 *>(codes + ((t0 + k) * per_token + c) * 8);
    const long long u = kvc_tok_unit(t0, m.tok_div) * m.sj + b * m.sb + h * m.sh + c0;
    const uint4 sv = *reinterpret_cast<const uint4 *>(m.scale + u);
    const __half2 *s2 = reinterpret_cast<const __half2 *>(&sv);
    const __half2 sc[4] = {s2[0], s2[1], s2[2], s2[3]};
    float mi[8];
    if (m.min_bytes == 1) {
        const uint2 mv = *reinterpret_cast<const uint2 *>(reinterpret_cast<const int8_t *>(m.min_int) + u);
        const int8_t *mb = reinterpret_cast<const int8_t *>(&mv);
#pragma unroll
        for (int k = 0; k < 8; k++) mi[k] = (float)mb[k] - 8388608.0f;
    } else {
        const uint4 mv = *reinterpret_cast<const uint4 *>(reinterpret_cast<const int16_t *>(m.min_int) + u);
        const int16_t *mh = reinterpret_cast<const int16_t *>(&mv);
#pragma unroll
        for (int k = 0; k < 8; k++) mi[k] = (float)mh[k] - 8388608.0f;
    }
#pragma unroll
    for (int k = 0; k < TOKENS; k++) *reinterpret_cast<uint4 *>(out + ((t0 + k) * per_token + c) * 8) = kvc_dequant8(cv[k].x, cv[k].y, mi, sc);
}
}  // namespace

extern "C" int kvc_dequant(const uint8_t *codes, const kvc_qmeta *q, int64_t T, int64_t B, int64_t H, int64_t D,
                           void *out, kvc_stream_t stream) {
    KVC_REQUIRE(codes && q && q->min_int && q->scale && out, "kvc_dequant: null pointer");
    KVC_REQUIRE(D > 0 && D % 8 == 0 && q->tok_div > 0, "kvc_dequant: bad shape");
    KVC_REQUIRE(q->min_bytes == 1 || q->min_bytes == 2, "kvc_dequant: min_bytes must be 1 or 2");
    long long rows = T * B * H, n = rows * (D / 8);
    if (n == 0) return KVC_OK;
    const kvc_qmeta_dev m = kvc_to_dev(*q);
    const int wide_units = m.sc == 1 && m.sj % 8 == 0 && m.sb % 8 == 0 && m.sh % 8 == 0 &&
                           (reinterpret_cast<uintptr_t>(m.scale) & 15) == 0 && (reinterpret_cast<uintptr_t>(m.min_int) & (8 * m.min_bytes - 1)) == 0;
    // (Four tokens and one per thread: 0.52 M values 2.04 and 2.04 us, 0.86 M 2.33 and 2.44, 1.05 M 2.34 and 2.75, 2.1 M 2.55 and 3.57, 8.4 M 5.0 and 8.7, 67 M 33 and
    // 56; 0.12 M 2.23 and 2.14, 0.26 M 2.04 and 1.94: below 512 threads per SM the single tokens fill the device better.)
    constexpr int TOKENS = 4;
    const long long per_token = B * H * (D / 8);
    if (wide_units && m.tok_div % TOKENS == 0 && T % TOKENS == 0 && n > 512ll * kvc_sm_count() && T / TOKENS <= 65535 && per_token < (1ll << 31)) {
        dequant_channel_kernel<TOKENS><<<dim3((unsigned)((per_token + 255) / 256), (unsigned)(T / TOKENS)), 256, 0, kvc_cu(stream)>>>(
            codes, m, (uint32_t)H, (uint32_t)(D / 8), (uint32_t)per_token, reinterpret_cast<__half *>(out));
        KVC_LAUNCH_OK();
        return KVC_OK;
    }
    const int groups = m.sc == 0 && n > 512ll * kvc_sm_count() ? 2 : 1;
    (groups == 2 ? dequant_kernel<2> : dequant_kernel<1>)<<<(unsigned)((n + 256 * groups - 1) / (256 * groups)), 256, 0, kvc_cu(stream)>>>(
        codes, m, rows, (uint32_t)B, (uint32_t)H, (uint32_t)D, wide_units, reinterpret_cast<__half *>(out));
    KVC_LAUNCH_OK();
    return KVC_OK;
}

extern "C" int kvc_k_matvec(const void *k, const void *q, void *out, int64_t ctx, int64_t H, kvc_stream_t stream) {
    KVC_REQUIRE(k && q && out, "kvc_k_matvec: null pointer");
    KVC_REQUIRE(ctx >= 0 && H > 0, "kvc_k_matvec: bad shape");
    long long rows = ctx * H;
    if (rows == 0) return KVC_OK;
    k_matvec_kernel<<<(unsigned)((rows + 7) / 8), 256, 0, kvc_cu(stream)>>>(
        reinterpret_cast<const __half *>(k), reinterpret_cast<const __half *>(q), reinterpret_cast<__half *>(out), rows, H);
    KVC_LAUNCH_OK();
    return KVC_OK;
}

// ---- rotary embedding of new keys on their way into the cache -------------------------------------
// models/cache/kvcomp_quant.py:43-48 rotates the new keys (utils/compute.py:25-33: t * cos + rotate_half(t) * sin,
// every op a rounded fp16 tensor op) before they enter the recent window; the cache keeps tokens token-major.
// One pass does both: x [B, H, t, D] -> out [t, B, H, D], same bits as torch's four ops and the transposing copy.
// blockIdx.y = 1 (kvc_kv_store): the same rows of a second tensor xv -> outv without rotation (the new values)
__global__ void __launch_bounds__(256) rope_store_kernel(const __half *__restrict__ x, const __half *__restrict__ cs,
                                                         const __half *__restrict__ sn, __half *__restrict__ out,
                                                         long long B, long long H, long long t, int D, long long cs_bstride, long long x_tokens,
                                                         const __half *__restrict__ xv, __half *__restrict__ outv) {
    // A kernel launched behind this one with programmatic stream serialisation (the fused attention, or its merge kernel
    // while nothing is compressed) may set up while these few rows are written: it touches them only after its own
    // grid-dependency wait.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (blockIdx.y == 1) { x = xv; out = outv; cs = nullptr; }
    const int per_row = D / 16;                                  // a thread: 8 channels of the lower half and their partners
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= t * B * H * per_row) return;
    const int c0 = (int)(i % per_row) * 8, half = D / 2;
    const long long row = i / per_row, h = row % H, b = (row / H) % B, tok = row / (H * B);
    const __half *xr = x + ((b * H + h) * x_tokens + tok) * D;
    __half *orow = out + ((tok * B + b) * H + h) * D;
    const uint4 xa = *reinterpret_cast<const uint4 *>(xr + c0), xb = *reinterpret_cast<const uint4 *>(xr + c0 + half);
    if (cs == nullptr) {                                         // no rotation (values): the transposition alone
        *reinterpret_cast<uint4 *>(orow + c0) = xa;
        *reinterpret_cast<uint4 *>(orow + c0 + half) = xb;
        return;
    }
    const __half *cr = cs + b * cs_bstride + tok * D, *sr = sn + b * cs_bstride + tok * D;
    const uint4 ca = *reinterpret_cast<const uint4 *>(cr + c0), cb = *reinterpret_cast<const uint4 *>(cr + c0 + half);
    const uint4 sa = *reinterpret_cast<const uint4 *>(sr + c0), sb = *reinterpret_cast<const uint4 *>(sr + c0 + half);
    uint4 oa, ob;
    rope8(xa, xb, ca, cb, sa, sb, oa, ob);
    *reinterpret_cast<uint4 *>(orow + c0) = oa;
    *reinterpret_cast<uint4 *>(orow + c0 + half) = ob;
}

// The same for a prompt (head_dim 128): a CTA takes 32 tokens of HT neighbouring heads.  rope_store_kernel's order, one row
// per head of a token, reads 256 bytes of a page at a time and fetches cos and sin for every head: 1 GiB of keys 515 us,
// and values went through torch's strided copy (1232 us).  Here a warp reads 1 KB runs of each head, writes runs of
// HT rows, and a thread keeps cos and sin over its heads and HT x 2 loads in flight: 349 and 320 us, the copy rate.  (HT = 2: 64
// registers, 40 bytes on the stack; 8 x 30 heads x 4096 tokens 91 and 78 us, the same bytes per us.)
template <int HT>
__global__ void __launch_bounds__(256) rope_tile_kernel(const __half *__restrict__ x, const __half *__restrict__ cs,
                                                        const __half *__restrict__ sn, __half *__restrict__ out,
                                                        uint32_t B, uint32_t H, long long t, long long cs_bstride, long long x_tokens) {
    const uint32_t groups = H / HT, b = blockIdx.x / groups, h0 = (blockIdx.x % groups) * HT;
    const long long tok = (long long)blockIdx.y * 32 + (threadIdx.x >> 3);
    const int c0 = (threadIdx.x & 7) * 8;
    if (tok >= t) return;
    const __half *xr = x + (((long long)b * H + h0) * x_tokens + tok) * 128 + c0;
    __half *orow = out + ((tok * B + b) * H + h0) * 128 + c0;
    uint4 xa[HT], xb[HT];
#pragma unroll
    for (int k = 0; k < HT; k++) {
        xa[k] = *reinterpret_cast<const uint4 *>(xr + k * x_tokens * 128);
        xb[k] = *reinterpret_cast<const uint4 *>(xr + k * x_tokens * 128 + 64);
    }
    if (cs != nullptr) {
        const __half *cr = cs + b * cs_bstride + tok * 128 + c0, *sr = sn + b * cs_bstride + tok * 128 + c0;
        const uint4 ca = *reinterpret_cast<const uint4 *>(cr), cb = *reinterpret_cast<const uint4 *>(cr + 64);
        const uint4 sa = *reinterpret_cast<const uint4 *>(sr), sb = *reinterpret_cast<const uint4 *>(sr + 64);
#pragma unroll
        for (int k = 0; k < HT; k++) { uint4 oa, ob; rope8(xa[k], xb[k], ca, cb, sa, sb, oa, ob); xa[k] = oa; xb[k] = ob; }
    }
#pragma unroll
    for (int k = 0; k < HT; k++) {
        *reinterpret_cast<uint4 *>(orow + k * 128) = xa[k];
        *reinterpret_cast<uint4 *>(orow + k * 128 + 64) = xb[k];
    }
}

extern "C" int kvc_rope_store_rows(const void *x, const void *cos_, const void *sin_, void *out, int64_t B, int64_t H, int64_t x_tokens,
                                   int64_t first, int64_t t, int64_t D, int64_t cos_batch_stride, kvc_stream_t stream) {
    KVC_REQUIRE(x && out && ((cos_ == nullptr) == (sin_ == nullptr)), "kvc_rope_store: null pointer");
    KVC_REQUIRE(B > 0 && H > 0 && t >= 0 && D > 0 && D % 16 == 0 && first >= 0 && first + t <= x_tokens, "kvc_rope_store: bad shape");
    KVC_REQUIRE(((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(cos_) | reinterpret_cast<uintptr_t>(sin_) |
                  reinterpret_cast<uintptr_t>(out)) & 15) == 0, "kvc_rope_store: pointers must be 16-byte aligned");
    KVC_REQUIRE(cos_batch_stride == 0 || cos_batch_stride == x_tokens * D, "kvc_rope_store: cos/sin must be [B, t, D] or [1, t, D]");
    const long long n = t * B * H * (D / 16);
    if (n == 0) return KVC_OK;
    KVC_REQUIRE((n + 255) / 256 < (1ll << 31), "kvc_rope_store: too many elements");
    const __half *xh = reinterpret_cast<const __half *>(x) + first * D;
    const __half *ch = cos_ ? reinterpret_cast<const __half *>(cos_) + first * D : nullptr, *sh = sin_ ? reinterpret_cast<const __half *>(sin_) + first * D : nullptr;
    __half *oh = reinterpret_cast<__half *>(out);
    // tiles when there are enough of them to fill the device twice over; else a thread per 16 channels of a row
    const int ht = H % 4 == 0 ? 4 : (H % 2 == 0 ? 2 : 1);
    const long long col_groups = B * (H / ht), tok_tiles = (t + 31) / 32;
    if (D == 128 && t >= 32 && col_groups * tok_tiles >= 2ll * kvc_sm_count() && tok_tiles <= 65535 && col_groups < (1ll << 31)) {
        auto *kernel = ht == 4 ? rope_tile_kernel<4> : (ht == 2 ? rope_tile_kernel<2> : rope_tile_kernel<1>);
        kernel<<<dim3((unsigned)col_groups, (unsigned)tok_tiles), 256, 0, kvc_cu(stream)>>>(xh, ch, sh, oh, (uint32_t)B, (uint32_t)H, t, cos_batch_stride, x_tokens);
        KVC_LAUNCH_OK();
        return KVC_OK;
    }
    rope_store_kernel<<<(unsigned)((n + 255) / 256), 256, 0, kvc_cu(stream)>>>(xh, ch, sh, oh, B, H, t, (int)D, cos_batch_stride, x_tokens, nullptr, nullptr);
    KVC_LAUNCH_OK();
    return KVC_OK;
}

extern "C" int kvc_rope_store(const void *x, const void *cos_, const void *sin_, void *out, int64_t B, int64_t H, int64_t t,
                              int64_t D, int64_t cos_batch_stride, kvc_stream_t stream) {
    return kvc_rope_store_rows(x, cos_, sin_, out, B, H, t, 0, t, D, cos_batch_stride, stream);
}

// Which prompts kvc_quantize_heads takes: K units per channel in blocks of 64 or 128 tokens; V units per token or vector, up to
// 64 heads (they are held in registers).  A unit must not span sequences.
extern "C" int kvc_quantize_heads_fits(int mode, int batch_shared, int64_t T, int64_t B, int64_t H, int64_t D, int64_t block) {
    if (D != 128 || B <= 0 || H <= 0 || B * H >= (1ll << 31) || T < 0) return 0;
    if (mode == KVC_MODE_CHANNEL) return (block == 64 || block == 128) && T / block <= 65535;
    if (mode == KVC_MODE_VECTOR) return H <= 64;
    return mode == KVC_MODE_TOKEN && H <= 64 && (!batch_shared || B == 1);
}

extern "C" int kvc_quantize_heads(const void *x, const void *cos_, const void *sin_, int64_t cos_batch_stride, int64_t B, int64_t H,
                                  int64_t x_tokens, int64_t T, int64_t D, int mode, int batch_shared, int64_t block, float rel,
                                  uint8_t *codes, void *min_int, int min_bytes, void *scale, unsigned long long *hist,
                                  int32_t *status, kvc_stream_t stream) {
    KVC_REQUIRE(x && codes && min_int && scale && status && (cos_ == nullptr) == (sin_ == nullptr), "kvc_quantize_heads: null pointer");
    KVC_REQUIRE(kvc_quantize_heads_fits(mode, batch_shared, T, B, H, D, block), "kvc_quantize_heads: these units take kvc_quantize");
    KVC_REQUIRE(T >= 0 && T <= x_tokens, "kvc_quantize_heads: %lld of %lld tokens", (long long)T, (long long)x_tokens);
    KVC_REQUIRE(min_bytes == 1 || min_bytes == 2, "kvc_quantize_heads: min_bytes must be 1 or 2");
    KVC_REQUIRE(cos_ == nullptr || mode == KVC_MODE_CHANNEL, "kvc_quantize_heads: only keys are rotated");
    KVC_REQUIRE(cos_batch_stride == 0 || cos_batch_stride == x_tokens * D, "kvc_quantize_heads: cos/sin must be [B, t, D] or [1, t, D]");
    KVC_REQUIRE(((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(cos_) | reinterpret_cast<uintptr_t>(sin_)) & 15) == 0 &&
                (reinterpret_cast<uintptr_t>(codes) & 7) == 0, "kvc_quantize_heads: x, cos and sin must be 16-byte and codes 8-byte aligned");
    if (T == 0) return KVC_OK;
    cudaStream_t s = kvc_cu(stream);
    const __half *xh = reinterpret_cast<const __half *>(x), *ch = reinterpret_cast<const __half *>(cos_), *sh = reinterpret_cast<const __half *>(sin_);
    __half *sc = reinterpret_cast<__half *>(scale);
    const long long sms = kvc_sm_count();
    if (mode == KVC_MODE_CHANNEL) {
        KVC_REQUIRE(T % block == 0, "kvc_quantize_heads: T=%lld is not a multiple of block=%lld", (long long)T, (long long)block);
        // heads per CTA: four share the reading of cos and sin, fewer where the device would not be full twice over
        long long heads = 4;
        while (heads > 1 && (T / block) * B * ((H + heads - 1) / heads) < 4 * sms) heads /= 2;
        // (two rows per thread: with one and twice the threads, a prompt of 32 x 4096 tokens, 1 GiB each of keys and
        // values, takes 2.94 ms instead of 2.48)
        auto *kernel = block == 64 ? (ch ? quant_heads_channel_kernel<2, 256, true> : quant_heads_channel_kernel<2, 256, false>)
                                   : (ch ? quant_heads_channel_kernel<2, 512, true> : quant_heads_channel_kernel<2, 512, false>);
        kernel<<<dim3((unsigned)(B * ((H + heads - 1) / heads)), (unsigned)(T / block)), block == 64 ? 256 : 512, 0, s>>>(
            xh, ch, sh, cos_batch_stride, (uint32_t)B, (uint32_t)H, (uint32_t)heads, x_tokens, rel, codes, min_int, min_bytes, sc, hist, status);
    } else {
        const long long groups = (T + 3) / 4 * B;
        const unsigned grid = (unsigned)std::min<long long>(groups, sms * 8);
#define KVC_QT(NH_) (mode == KVC_MODE_VECTOR ? quant_heads_token_kernel<NH_, true> : quant_heads_token_kernel<NH_, false>)<<<grid, 256, 0, s>>>( \
        xh, (uint32_t)B, (uint32_t)H, x_tokens, T, rel, codes, min_int, min_bytes, sc, hist, status)
        if (H <= 4) KVC_QT(1);
        else if (H <= 8) KVC_QT(2);
        else if (H <= 16) KVC_QT(4);
        else if (H <= 32) KVC_QT(8);
        else KVC_QT(16);
#undef KVC_QT
    }
    KVC_LAUNCH_OK();
    return KVC_OK;
}

extern "C" int kvc_kv_store(const void *k, const void *v, const void *cos_, const void *sin_, void *kout, void *vout,
                            int64_t B, int64_t H, int64_t t, int64_t D, int64_t cos_batch_stride, kvc_stream_t stream) {
    KVC_REQUIRE(k && v && cos_ && sin_ && kout && vout, "kvc_kv_store: null pointer");
    KVC_REQUIRE(B > 0 && H > 0 && t >= 0 && D > 0 && D % 16 == 0, "kvc_kv_store: bad shape");
    KVC_REQUIRE(((reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(cos_) |
                  reinterpret_cast<uintptr_t>(sin_) | reinterpret_cast<uintptr_t>(kout) | reinterpret_cast<uintptr_t>(vout)) & 15) == 0,
                "kvc_kv_store: pointers must be 16-byte aligned");
    KVC_REQUIRE(cos_batch_stride == 0 || cos_batch_stride == t * D, "kvc_kv_store: cos/sin must be [B, t, D] or [1, t, D]");
    const long long n = t * B * H * (D / 16);
    if (n == 0) return KVC_OK;
    KVC_REQUIRE((n + 255) / 256 < (1ll << 31), "kvc_kv_store: too many elements");
    rope_store_kernel<<<dim3((unsigned)((n + 255) / 256), 2), 256, 0, kvc_cu(stream)>>>(
        reinterpret_cast<const __half *>(k), reinterpret_cast<const __half *>(cos_), reinterpret_cast<const __half *>(sin_),
        reinterpret_cast<__half *>(kout), B, H, t, (int)D, cos_batch_stride, t,
        reinterpret_cast<const __half *>(v), reinterpret_cast<__half *>(vout));
    KVC_LAUNCH_OK();
    return KVC_OK;
}

extern "C" int kvc_kv_store_packed(const kvc_kv_store_args *args, kvc_stream_t stream) {
    KVC_REQUIRE(args, "kvc_kv_store_packed: null pointer");
    kvc_kv_store_args a;
    memcpy(&a, args, sizeof(a));                                // (wherever the caller packed them)
    return kvc_kv_store(a.k, a.v, a.cos_, a.sin_, a.kout, a.vout, a.B, a.H, a.t, a.D, a.cos_batch_stride, stream);
}

// ---- the quantiser in two calls: extremes first, codes later --------------------------------------
// For units made of whole (token, sequence) rows -- BlockQuant and TokenQuant, whose units span the heads
// (models/cache/kvcomp_encode.py:10-13, utils/compute.py:138-143).  When the heads of a cache are split
// over several GPUs, every rank takes the extremes of its own heads, the ranks exchange them (elementwise
// min and max), and every rank quantises with the joint extremes: same scale, min_int and codes as one GPU
// holding all heads would produce.
static int ranged_units(int mode, int batch_shared, int64_t T, int64_t B, int64_t block, long long *n_units, int *tok_div) {
    KVC_REQUIRE(mode == KVC_MODE_BLOCK || mode == KVC_MODE_TOKEN, "units of mode %d do not span heads: use kvc_quantize", mode);
    if (mode == KVC_MODE_BLOCK) KVC_REQUIRE(block > 0 && T % block == 0, "T=%lld is not a multiple of block=%lld", (long long)T, (long long)block);
    *tok_div = mode == KVC_MODE_BLOCK ? (int)block : 1;
    *n_units = (T / *tok_div) * (batch_shared ? 1 : B);
    return KVC_OK;
}

extern "C" int kvc_quant_minmax(const void *x, int64_t T, int64_t B, int64_t H, int64_t D, int mode, int batch_shared,
                                int64_t block, void *mn_out, void *mx_out, void *workspace, int64_t workspace_bytes,
                                kvc_stream_t stream) {
    KVC_REQUIRE(x && mn_out && mx_out, "kvc_quant_minmax: null pointer");
    KVC_REQUIRE(T >= 0 && B > 0 && H > 0 && D > 0 && (H * D) % 8 == 0, "kvc_quant_minmax: bad shape");
    KVC_REQUIRE((reinterpret_cast<uintptr_t>(x) & 15) == 0, "kvc_quant_minmax: x must be 16-byte aligned");
    long long n_units; int tok_div;
    if (int rc = ranged_units(mode, batch_shared, T, B, block, &n_units, &tok_div)) return rc;
    if (T == 0) return KVC_OK;
    KVC_REQUIRE(workspace && workspace_bytes >= n_units * 8, "kvc_quant_minmax: needs %lld bytes of workspace", n_units * 8);
    KVC_REQUIRE(T * B < (1ll << 31), "kvc_quant_minmax: too many rows");
    cudaStream_t s = kvc_cu(stream);
    unsigned int *ws = reinterpret_cast<unsigned int *>(workspace);
    KVC_CUDA_OK(cudaMemsetAsync(ws, 0, n_units * 8, s));
    quant_block_minmax_kernel<<<(unsigned)(T * B), 256, 0, s>>>(reinterpret_cast<const __half *>(x), B, H * D, tok_div, batch_shared, ws);
    quant_minmax_export_kernel<<<(unsigned)((n_units + 127) / 128), 128, 0, s>>>(ws, n_units, reinterpret_cast<__half *>(mn_out),
                                                                                  reinterpret_cast<__half *>(mx_out));
    KVC_LAUNCH_OK();
    return KVC_OK;
}

extern "C" int kvc_quantize_ranged(const void *x, int64_t T, int64_t B, int64_t H, int64_t D, int mode, int batch_shared,
                                   int64_t block, float rel, const void *mn_in, const void *mx_in,
                                   uint8_t *codes, void *min_int, int min_bytes, void *scale, unsigned long long *hist,
                                   void *workspace, int64_t workspace_bytes, int32_t *status, kvc_stream_t stream) {
    KVC_REQUIRE(x && mn_in && mx_in && codes && min_int && scale && status, "kvc_quantize_ranged: null pointer");
    KVC_REQUIRE(T >= 0 && B > 0 && H > 0 && D > 0 && (H * D) % 8 == 0, "kvc_quantize_ranged: bad shape");
    KVC_REQUIRE(min_bytes == 1 || min_bytes == 2, "kvc_quantize_ranged: min_bytes must be 1 or 2");
    KVC_REQUIRE((reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(codes) & 7) == 0,
                "kvc_quantize_ranged: x must be 16-byte and codes 8-byte aligned");
    long long n_units; int tok_div;
    if (int rc = ranged_units(mode, batch_shared, T, B, block, &n_units, &tok_div)) return rc;
    if (T == 0) return KVC_OK;
    KVC_REQUIRE(workspace && workspace_bytes >= n_units * 8, "kvc_quantize_ranged: needs %lld bytes of workspace", n_units * 8);
    KVC_REQUIRE(T * B < (1ll << 31), "kvc_quantize_ranged: too many rows");
    cudaStream_t s = kvc_cu(stream);
    unsigned int *ws = reinterpret_cast<unsigned int *>(workspace);
    quant_block_finalize_kernel<<<(unsigned)((n_units + 127) / 128), 128, 0, s>>>(
        ws, n_units, rel, min_int, min_bytes, reinterpret_cast<__half *>(scale), status,
        reinterpret_cast<const __half *>(mn_in), reinterpret_cast<const __half *>(mx_in));
    quant_block_apply_kernel<<<(unsigned)(T * B), 256, 0, s>>>(reinterpret_cast<const __half *>(x), B, H * D, tok_div, batch_shared,
                                                               ws, codes, hist, status);
    KVC_LAUNCH_OK();
    return KVC_OK;
}
