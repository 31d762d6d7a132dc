// Fused decompress + mat-vec kernels: q.K^T scores, P.V partials, and the one-pass decode
// attention (q.K^T -> online softmax -> P.V) straight from the compressed streams.
//
// Reference kernels restated: huffman_decode_and_mat_vec_mul (kernels.cu:721-776),
// v_huffman_decode_and_mat_vec_mul (kernels.cu:778-861); attention semantics of
// eager_attention_forward (models/llama.py:211-234).
//
// Work layout of the unfused kernels: CTA = 256 threads working on 256 tokens of one (b, kv head); of the attention kernels: a
// worker of 128 threads, several to a CTA, walking steps of 128 tokens.
//   K phase: thread = token; its vector holds the token's 128 channel codes.
//            score = sum_c code_c * w[c] + zp, with w[c] = q[c]*scale[c] staged per 64-token block
//            (dequantisation folded into the weights, the min_int term summed once per block).
//   V phase: thread = (128-token group, channel); its vector holds 128 tokens of that channel.
//            out[ch] = sum_t code_t * ps[t] + zpv, with ps[t] = p[t]*scale[t] staged per group.
// The attention kernels are launched with as many workers as the device holds at once.  Their work is cut into
// items (one (b, kv head) column x one run of steps); a worker starts with items fixed by its index and draws the rest
// from a counter, so that the workers an SM's schedulers favour take more of them: with one head per KV head two fixed and
// two ahead, with several one fixed and one ahead.  Staging copies, a step's metadata and the query vector of the next step or
// item are always fetched while the current one is decoded.  When a column has more than one item,
// each leaves a partial result (max, sum, accumulators) and a second kernel merges them.
// Both phases are "decode 128 symbols and dot them with a shared 128-vector", so they share one
// decoder.  The shared vector is held in 16-bit block fixed point, one fp32 step per vector; the products with the symbols are integer arithmetic,
// exact, accumulated in int32.  The only rounding is that of the weights (2^-16 of the largest weight of the vector); the zero-point terms and
// everything after the dot product are fp32.  In the unfused kernels and with one head per KV head a weight is step * (256*hi + lo), hi a signed and
// lo an unsigned byte: every table lookup yields up to three symbols as bytes, and two dp4a instructions multiply them with the matching weight
// bytes.  With several query heads per KV head they share every decode: in the unfused kernels by weight records [position][G], up to four heads
// a launch, in the attention kernel by matrix instructions with both bytes signed (attn_rows_kernel).
#include <math_constants.h>
#include <string.h>

#include <algorithm>
#include <type_traits>

#include "kvc_decode.cuh"

namespace {

constexpr int SLOT_PAD = 1024;           // readable bytes behind the last staging slot
constexpr int NTHR = 256;
constexpr size_t MAX_CTA_SHARED = 227 * 1024;
constexpr int ATTN_PART_FLOATS = 4 + 256;   // workspace per head and run of 256-token tiles: two partial results (ROWS_PART_FLOATS each)

struct CacheDev {
    const uint8_t *encoded;
    long long encoded_bytes;
    const uint2 *block_info;
    const uint16_t *thread_info;
    const void *book;
    kvc_qmeta_dev q;
    uint32_t max_block;           // upper bound of a block's byte count
};

// a staging slot holds the largest block plus its alignment lead, widened to 16-byte chunks, plus the decoder's two words
// of read-ahead
__host__ __device__ __forceinline__ uint32_t slot_bytes_of(uint32_t max_block) { return ((max_block + 15u + 15u) & ~15u) + 16u; }

CacheDev to_dev(const kvc_cache &c) {
    CacheDev d;
    d.max_block = (c.max_block_bytes > 0 && c.max_block_bytes < 8191) ? (uint32_t)c.max_block_bytes : 8191u;
    d.encoded = c.encoded; d.encoded_bytes = c.encoded_bytes;
    d.block_info = reinterpret_cast<const uint2 *>(c.block_info); d.thread_info = c.thread_info;
    d.book = c.book; d.q = kvc_to_dev(c.q);
    return d;
}

// ---- 16-bit fixed-point weight records -----------------------------------------------------------
// per position c: a word {0, hi(w[c]), hi(w[c+1]), hi(w[c+2])} and a word of the lo bytes laid out the
// same way, so that a decode-table entry {advance, s0, s1, s2} multiplies them directly (the advance
// byte meets the zero).  pack4 gives {hi word, lo word}; q3 is unused.
__device__ __forceinline__ uint2 pack4(int q0, int q1, int q2, int /*q3*/) {
    uint2 r;
    r.x = (((uint32_t)(q0 >> 8) & 0xffu) << 8) | (((uint32_t)(q1 >> 8) & 0xffu) << 16) | (((uint32_t)(q2 >> 8) & 0xffu) << 24);
    r.y = (((uint32_t)q0 & 0xffu) << 8) | (((uint32_t)q1 & 0xffu) << 16) | (((uint32_t)q2 & 0xffu) << 24);
    return r;
}
__device__ __forceinline__ float fix_step(float wmax) { return wmax > 0.f ? wmax * (1.0f / 32767.0f) : 0.f; }
__device__ __forceinline__ int fix_quant(float w, float step) { return step > 0.f ? __float2int_rn(w / step) : 0; }
__device__ __forceinline__ float fix_value(float step, int hi, int lo) { return step * fmaf((float)hi, 256.0f, (float)lo); }

__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}

// ---- grouped queries (the attention kernel, G >= 2): decode first, multiply on the tensor cores -------
// With several query heads per KV head the weight records of a position grow to 16 bytes and more, and 32
// lanes at 32 different positions fetch 0.5 KB and more per lookup: the kernel becomes bound by shared-memory
// wavefronts.  So a warp decodes 32 symbols of each of its 32 vectors into rows of bytes in shared memory (KvcCursor: every lane
// at the same position), and m16n8k32 integer instructions multiply the rows with the weights: two columns per head, the hi and
// the lo bytes.  The integer sums are the same as in the one-pass form.  What bounds it: the shared-memory pipe (849 wavefronts per warp
// and step of 128 tokens, 76 % busy; nine per round of two lookups) and, with 2610 instructions, issue (59 %) together.  One layer of
// 16 sequences x 32768 tokens, 8 x 4 heads, rel 0.05 / 0.1: whole rows, each lane at its own position, up to three symbols per lookup (3440 instructions,
// 1010 wavefronts) 650 us, now 536; 32 x 16384 tokens, 10 x 4, rel 0.02 / 0.15, 868 and 835; 4096 tokens of the first, 104 and 88.  (In an earlier state six workers
// of 80 registers took 562 to 576 us where five of 96 took 577; tables of 8 to 12 bits repeated over the banks, 32 KB each, one symbol per lookup, 660.)
constexpr int WROW = 136;                 // weight words per vector of the one-pass form: 128 positions + zeroed overrun

// Rows of 32 symbols, two units of 16 bytes each, swapped in every other four rows: a quarter warp's stores (eight rows, one unit) and a half
// warp's loads (four rows, 8 bytes a lane) then meet every bank once.  32 symbols are one k step of the matrix instruction:
// the rows of a warp take 1 KB instead of 4.5.
constexpr int ROW_BYTES = 32;
// A brief launch (two steps per worker, one after the other, at most) is a matter of latency: its vectors are decoded whole, with up to three symbols per lookup and no
// table to be made first, into rows of 128 symbols, the overrun of paired lookups and a 16-byte alignment that spreads over the banks.  (Device time by pairs or
// singles, and whole: 2 columns of 8192 tokens, 4 heads, 16.5 and 13.3 us; 128 columns of 512, 22.0 and 20.8, of 768, two steps per worker, 31.2 and 29.4,
// at rel 0.02 / 0.02 38.5 and 33.3; of 1536, three steps, 45.5 either way; without a workspace 32 columns of 2048, four steps, 48.0 and 49.1, 8 of 8192 147 and 157.)
constexpr int BRIEF_STEPS = 2;
constexpr int WHOLE_ROW_BYTES = 144;
static_assert(WHOLE_ROW_BYTES >= 128 + KVC_DECODE_OVERRUN + 3, "rows too short for paired lookups");
// A vector's weights: two columns per head, the hi and the lo bytes of 4 positions to a word.  Column stride 40 words: the fragment
// loads (four columns x 32 bytes per half warp) meet every bank once.
constexpr int COL_WORDS = 40;
__host__ __device__ constexpr int vec_words(int G) { return 2 * G * COL_WORDS; }
// 16-bit fixed point as two signed bytes (value = step * (256 * hi + lo)): -128 * 257 .. 127 * 257.
// K's weights: the larger sign takes the negative side, to -32767.  Where the largest of the other sign is within 0.4 % of it, that one takes 32639, and the
// step is up to 0.4 % coarser than in a symmetric range.
constexpr float FIX_DOWN = 32767.0f, FIX_UP = 32639.0f;
// V's weights: the largest one is 1 and takes 32880 (below the end, 32896, by what the approximate logarithm and power can be off together).
// Their reference is a score plus a logarithm, rounded up: below FAR that lowers them by a factor of exp(-2^-9) at most, and the fixed-point step stays
// finer than 1/32767 of the largest.  Beyond FAR the reference is the largest score itself, and the largest weight is looked for.
constexpr float FIX_V = 32880.0f, FAR = 32768.0f;
constexpr float LOG2E = 1.4426950408889634f, LN2 = 0.6931471805599453f;
// (Scores stay in units of e, as the merge kernel and the dense rows behind the compressed part have them: a factor of log2 e in the query would round every
// score, and at 1e4 two equal ones by two ways weigh 1e-3 apart.)
__device__ __forceinline__ float exp_fast(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x * LOG2E)); return y; }
__device__ __forceinline__ float log2_fast(float x) { float y; asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ float rcp_fast(float x) { float y; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }

// {hi word, lo word} of four values times inv, all of them within the range.  The product is rounded by adding 1.5 * 2^23, whose low bits
// then hold it, and 128 more: byte 1 is the hi byte, byte 0 the lo byte with its sign bit turned.
__device__ __forceinline__ uint2 pack_fix(float a, float b, float c, float d, float inv) {
    const uint32_t t0 = __float_as_uint(fmaf(a, inv, 12583040.0f)), t1 = __float_as_uint(fmaf(b, inv, 12583040.0f));
    const uint32_t t2 = __float_as_uint(fmaf(c, inv, 12583040.0f)), t3 = __float_as_uint(fmaf(d, inv, 12583040.0f));
    const uint32_t x = __byte_perm(t0, t1, 0x5140), y = __byte_perm(t2, t3, 0x5140);          // {lo0, lo1, hi0, hi1}
    return make_uint2(__byte_perm(x, y, 0x7632), __byte_perm(x, y, 0x5410) ^ 0x80808080u);
}

// c += A (16 x 32 unsigned bytes) * B (32 x 8 signed bytes)
__device__ __forceinline__ void mma_us(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint2 b) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b.x), "r"(b.y));
}
__device__ __forceinline__ void sts128(uint32_t addr, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" :: "r"(addr), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

// Which of its warp's 32 vectors a lane decodes.  Rows r, r + 8, r + 16 and r + 24 of a warp's matrix end up in the lanes 4 r .. 4 r + 3: with
// this order they are the vectors 4 r .. 4 r + 3, four neighbouring tokens or channels.
__device__ __forceinline__ int vec_of_lane(int lane) { return 4 * (lane & 7) + (lane >> 3); }

// Decode a warp's 32 vectors, 32 symbols at a time, and multiply them with the weight columns at shared address w_s.  d[i][j]: vector
// 4 * (lane >> 2) + i, head (lane & 3) % G + 4 * j.  A lane's two columns of the product are the hi and the lo sums of its head, so they
// meet without an exchange; which word is which k index is free as long as A and B agree: a lane reads 8 consecutive bytes.
// (A column of hi bytes per head in one matrix instruction and one of lo bytes in another, the rows whole and decoded with up to three
// symbols per lookup at places of their own: twice the matrix instructions, twice the values per lane behind them with four heads.)
template <int G> struct RowsSum {
    static constexpr int HL = G == 8 ? 2 : 1;                  // heads per lane
    int c[HL][2][4];
    __device__ __forceinline__ RowsSum() {
#pragma unroll
        for (int j = 0; j < HL; j++)
#pragma unroll
            for (int t = 0; t < 2; t++)
#pragma unroll
                for (int i = 0; i < 4; i++) c[j][t][i] = 0;
    }
    // 32 symbols: get: the lane's place in row lane >> 2; rows lie `stride` bytes apart; col: its place in its weight column
    __device__ __forceinline__ void add(uint32_t get, uint32_t stride, uint32_t col) {
        const uint2 a0 = kvc_lds64(get), a1 = kvc_lds64(get + 8 * stride), a2 = kvc_lds64(get + 16 * stride), a3 = kvc_lds64(get + 24 * stride);
#pragma unroll
        for (int j = 0; j < HL; j++) {
            const uint2 bw = kvc_lds64(col + j * (8 * COL_WORDS * 4));
            mma_us(c[j][0], a0.x, a1.x, a0.y, a1.y, bw);
            mma_us(c[j][1], a2.x, a3.x, a2.y, a3.y, bw);
        }
    }
    __device__ __forceinline__ void out(int (&d)[4][HL]) const {
#pragma unroll
        for (int j = 0; j < HL; j++) {                         // |256 hi + lo| <= 128 * 255 * 32896 < 2^31
            d[0][j] = 256 * c[j][0][0] + c[j][0][1]; d[1][j] = 256 * c[j][0][2] + c[j][0][3];
            d[2][j] = 256 * c[j][1][0] + c[j][1][1]; d[3][j] = 256 * c[j][1][2] + c[j][1][3];
        }
    }
};
// What a vector is decoded from: shared addresses of its slot, the table (of single symbols: lone) and the tree.  (Both tables' addresses are the same for the
// whole launch: one that is chosen from step to step costs an addition per lookup, 2 % of the kernel's time.)
struct RowsFrom { uint32_t slot, at, lut, lone, tree; };

// lagged: in how many of the four parts a lane fell too far behind for PAIRS' rounds.
template <int G, int WAY, bool ESC>
__device__ __forceinline__ bool rows_dot_way(const RowsFrom &f, uint32_t rows_s, uint32_t w_s, int lane, int (&d)[4][RowsSum<G>::HL], uint32_t &lagged) {
    const uint32_t r = lane >> 2, q = lane & 3;
    const uint32_t put = rows_s + lane * ROW_BYTES + (r & 1u) * 16;
    const uint32_t get = rows_s + r * ROW_BYTES + (((q >> 1) ^ (r >> 2 & 1u)) * 16) + (q & 1u) * 8;
    const uint32_t col = w_s + (r % (2 * G)) * (COL_WORDS * 4) + q * 8;
    KvcCursor at(f.slot, f.at);
    RowsSum<G> sum;
    auto word = [&](bool end) { return WAY == KVC_PAIRS ? at.pairs<ESC>(f.lut, f.tree, end) : at.singles<ESC>(f.lone, f.tree); };
    if (WAY == KVC_PAIRS) word(false);
#pragma unroll 1
    for (uint32_t ch = 0; ch < 4; ch++) {
        const uint32_t s0 = at.s, ptr0 = at.ptr, last0 = at.last, behind0 = at.behind;
#pragma unroll ESC ? 1 : 2
        for (uint32_t u = 0; u < 2; u++) {
            const uint32_t w0 = word(false), w1 = word(false), w2 = word(false), w3 = word(ch + u == 4u);
            sts128(u ? put ^ 16u : put, w0, w1, w2, w3);
        }
        if (WAY == KVC_PAIRS && __any_sync(0xffffffffu, at.behind >= 24u)) {
            // a lane that fell more than a word behind takes the 32 symbols again; it and the others that are behind catch up
            lagged += __any_sync(0xffffffffu, at.behind > 32u);
            if (at.behind > 32u)
                at.again<ESC>(f.lut, f.tree, s0, ptr0, last0, behind0, ch == 3, [&](uint32_t k, uint32_t w) { asm volatile("st.shared.u32 [%0], %1;" :: "r"((k < 4 ? put : put ^ 16u) + (k & 3u) * 4), "r"(w) : "memory"); });
            if (ch < 3) at.catch_up<ESC>(f.lut, f.tree);
        }
        __syncwarp();
        sum.add(get, ROW_BYTES, col + ch * 32);
        __syncwarp();
    }
    sum.out(d);
    return at.ok;
}
// a vector at a time, each lane at its own place, into whole rows
template <int G, bool ESC>
__device__ __forceinline__ bool rows_dot_whole(const RowsFrom &f, uint32_t rows_s, uint32_t w_s, int lane, int (&d)[4][RowsSum<G>::HL]) {
    const uint32_t r = lane >> 2, q = lane & 3;
    KvcRowWriter put;
    const bool ok = kvc_decode_vector<ESC, 0>(f.slot, f.at, f.lut, KvcTreeShared{f.tree}, rows_s + lane * WHOLE_ROW_BYTES, put);
    __syncwarp();
    RowsSum<G> sum;
#pragma unroll
    for (uint32_t ch = 0; ch < 4; ch++) sum.add(rows_s + r * WHOLE_ROW_BYTES + ch * 32 + q * 8, WHOLE_ROW_BYTES, w_s + (r % (2 * G)) * (COL_WORDS * 4) + ch * 32 + q * 8);
    __syncwarp();
    sum.out(d);
    return ok;
}
template <int G>
__device__ __forceinline__ bool rows_dot(const KvcWay &way, const RowsFrom &f, uint32_t rows_s, uint32_t w_s, int lane, int (&d)[4][RowsSum<G>::HL], uint32_t &lagged) {
    if (way.way == KVC_WHOLE) return way.esc ? rows_dot_whole<G, true>(f, rows_s, w_s, lane, d) : rows_dot_whole<G, false>(f, rows_s, w_s, lane, d);
    if (!way.esc) return way.way == KVC_PAIRS ? rows_dot_way<G, KVC_PAIRS, false>(f, rows_s, w_s, lane, d, lagged) : rows_dot_way<G, KVC_SINGLES, false>(f, rows_s, w_s, lane, d, lagged);
    return way.way == KVC_PAIRS ? rows_dot_way<G, KVC_PAIRS, true>(f, rows_s, w_s, lane, d, lagged) : rows_dot_way<G, KVC_SINGLES, true>(f, rows_s, w_s, lane, d, lagged);
}

// Where the hi / lo weight word of position c and head g sits in a vector's 2 * WROW * G words.  One or
// two heads: a record {hi[G], lo[G]} per position, fetched with one 8- or 16-byte load.  Four heads: all
// hi records, then all lo records (16 bytes each), because 32-byte records would leave half of the banks idle.
template <int G> __device__ __forceinline__ constexpr int w_hi(int c, int g) { return G == 4 ? c * 4 + g : c * 2 * G + g; }
template <int G> __device__ __forceinline__ constexpr int w_lo(int c, int g) { return G == 4 ? WROW * 4 + c * 4 + g : c * 2 * G + G + g; }

// decode the thread's vector (staged at shared address slot_s) and dot it with the weight records at
// shared address w_s (layout: w_hi / w_lo)
template <int G, bool ESC, class Tree>
__device__ __forceinline__ bool decode_dot_impl(uint32_t slot_s, uint32_t byte_pos, uint32_t lut_s, Tree tree,
                                                uint32_t w_s, int (&hi)[G], int (&lo)[G]) {
    constexpr int SHIFT = G == 1 ? 3 : 4;                      // log2 of the record's bytes
    auto emit = [&](uint32_t syms, uint32_t a, uint32_t, uint32_t) {
        if (G == 4) {
            const uint4 x = lds128(a), y = lds128(a + WROW * 16);
            hi[0] = kvc_dp4a_us(syms, x.x, hi[0]); lo[0] = kvc_dp4a_uu(syms, y.x, lo[0]);
            hi[1 % G] = kvc_dp4a_us(syms, x.y, hi[1 % G]); lo[1 % G] = kvc_dp4a_uu(syms, y.y, lo[1 % G]);
            hi[2 % G] = kvc_dp4a_us(syms, x.z, hi[2 % G]); lo[2 % G] = kvc_dp4a_uu(syms, y.z, lo[2 % G]);
            hi[3 % G] = kvc_dp4a_us(syms, x.w, hi[3 % G]); lo[3 % G] = kvc_dp4a_uu(syms, y.w, lo[3 % G]);
        } else if (G == 2) {
            const uint4 x = lds128(a);
            hi[0] = kvc_dp4a_us(syms, x.x, hi[0]); lo[0] = kvc_dp4a_uu(syms, x.z, lo[0]);
            hi[1 % G] = kvc_dp4a_us(syms, x.y, hi[1 % G]); lo[1 % G] = kvc_dp4a_uu(syms, x.w, lo[1 % G]);
        } else {
            const uint2 x = kvc_lds64(a);
            hi[0] = kvc_dp4a_us(syms, x.x, hi[0]);
            lo[0] = kvc_dp4a_uu(syms, x.y, lo[0]);
        }
    };
    // two lookups per round: the weight rows keep WROW - 128 zeroed positions for what is emitted past 127
    static_assert(WROW >= 128 + KVC_DECODE_OVERRUN + 1, "weight rows too short for paired lookups");
    return kvc_decode_vector<ESC, SHIFT>(slot_s, byte_pos, lut_s, tree, w_s >> SHIFT, emit);
}
// esc: the book has codes longer than the table window (uniform over the CTA)
template <int G>
__device__ __forceinline__ bool decode_dot(const uint8_t *slot, uint32_t byte_pos, const KvcBookSmem &book, bool esc,
                                           const uint32_t *w, int (&hi)[G], int (&lo)[G]) {
    const uint32_t slot_s = kvc_smem_addr(slot), lut_s = kvc_smem_addr(book.lut), tree_s = kvc_smem_addr(book.tree),
                   w_s = kvc_smem_addr(w);
    return esc ? decode_dot_impl<G, true>(slot_s, byte_pos, lut_s, KvcTreeShared{tree_s}, w_s, hi, lo)
               : decode_dot_impl<G, false>(slot_s, byte_pos, lut_s, KvcTreeShared{tree_s}, w_s, hi, lo);
}
__device__ __forceinline__ bool book_has_long_codes(const void *book) {
    return kvc_book_needs_escape(book);
}

// ---- staging --------------------------------------------------------------------------------------
// plain loads: the 64 threads of a sub-group copy block `blk` into `slot`
// *nb receives the block's byte count: a vector that starts at or beyond it is not decoded
__device__ __forceinline__ bool stage(const CacheDev &kc, long long blk, uint8_t *slot, uint32_t *lead, uint32_t *nb, int v) {
    const uint2 bi = kc.block_info[blk];
    const uint32_t nbytes = bi.y & 0xffffu;
    *nb = nbytes;
    if (nbytes == 0 || nbytes > kc.max_block || (long long)bi.x + nbytes > kc.encoded_bytes) { *lead = 0; *nb = 0; return false; }
    *lead = kvc_stage_block(slot, kc.encoded, kc.encoded_bytes, bi.x, nbytes, v, 64);
    return true;
}

// bulk copies: lane `l` (< 4) of one warp issues the copy of its block; the whole warp must call.
// The source range is widened to 16-byte boundaries; `encoded` is 16-byte aligned and readable to
// the next boundary past its end (checked / required by the host code).
// starve (tests of the bounded waits only): announce 16 bytes and copy nothing, so that the phase never
// completes and nothing is in flight when the waiting threads give up.
__device__ __forceinline__ void stage_bulk(const CacheDev &kc, bool valid, long long blk, uint8_t *slot,
                                           uint32_t *lead, int *ok, uint32_t *nb, uint64_t *bar, int lane, bool starve = false) {
    uint32_t bytes = 0, ld = 0, nbytes = 0;
    const uint8_t *a0 = nullptr;
    bool good = false;
    if (lane < 4 && valid) {
        const uint2 bi = kc.block_info[blk];
        nbytes = bi.y & 0xffffu;
        good = nbytes != 0 && nbytes <= kc.max_block && (long long)bi.x + nbytes <= kc.encoded_bytes;
        if (good) {
            const uint8_t *src = kc.encoded + bi.x;
            ld = (uint32_t)(reinterpret_cast<uintptr_t>(src) & 15);
            a0 = src - ld;
            bytes = (ld + nbytes + 15u) & ~15u;
        }
    }
    if (starve) bytes = 0;
    uint32_t total = bytes;
    total += __shfl_xor_sync(0xffffffffu, total, 1);
    total += __shfl_xor_sync(0xffffffffu, total, 2);
    if (lane == 0) kvc_mbar_expect_tx(bar, starve ? 16u : total);   // one arrival per phase, even for 0 bytes
    __syncwarp();
    if (lane < 4) {
        lead[lane] = ld; ok[lane] = good; nb[lane] = good ? nbytes : 0u;
        if (bytes) kvc_bulk_g2s(slot, a0, bytes, bar);
    }
}

__device__ __forceinline__ uint32_t vec_start(const uint16_t *thread_info, long long blk, int v) {
    return v ? (uint32_t)(thread_info[blk * 64 + v - 1] >> 3) : 0u;
}
// the same in two steps: the load (issued a tile ahead) and the shift (at the use)
__device__ __forceinline__ unsigned short vec_start_bits(const uint16_t *thread_info, long long blk, int v) {
    unsigned short r = 0;
    if (v) r = thread_info[blk * 64 + v - 1];
    return r;
}

__device__ __forceinline__ unsigned short vec_start_bits32(const uint16_t *thread_info, uint32_t blk, int v) {
    return v ? thread_info[(size_t)blk * 64 + (uint32_t)(v - 1)] : (unsigned short)0;
}
// unit j of (sequence, head): what kvc_qmeta says, the channel aside
__device__ __forceinline__ long long unit_of(const kvc_qmeta_dev &m, uint32_t j, int b, int h) {
    return (long long)((unsigned long long)j * (unsigned long long)m.sj + (unsigned long long)(uint32_t)b * (unsigned long long)m.sb + (unsigned long long)(uint32_t)h * (unsigned long long)m.sh);
}

// ---- K weights --------------------------------------------------------------------------------------
// Weight records of the 4 blocks of a 256-token tile: w[sub][c][hi|lo][g], step[sub][g], zp[sub][g].
// Warp `wp` owns block sub = wp & 3 and the query heads g = (wp >> 2) * GH .. + GH - 1 (GH = G/2, or
// all of them on warps 0-3 when G = 1); lane = 4 consecutive channels.
// Units that depend on the channel (sc != 0) need tok_div % 64 == 0 so that a block shares them;
// otherwise scale and min_int are per-token scalars applied after the dot product (k_finish).
// scale (fp16 bits) and min_int of the lane's 4 consecutive channels, as two vector loads leave them: no
// arithmetic touches the words before their use, and they occupy 3 or 4 registers instead of 8
struct KUnit { uint2 sc; uint2 mi; };
__device__ __forceinline__ unsigned short ku_scale(const KUnit &u, int i) {
    const uint32_t w = i < 2 ? u.sc.x : u.sc.y;
    return (unsigned short)((i & 1) ? (w >> 16) : (w & 0xffffu));
}
__device__ __forceinline__ int ku_min(const KUnit &u, int i, int min_bytes) {
    if (min_bytes == 1) return (int)(signed char)((u.mi.x >> (8 * i)) & 0xffu);
    const uint32_t w = i < 2 ? u.mi.x : u.mi.y;
    return (int)(short)((i & 1) ? (w >> 16) : (w & 0xffffu));
}

// global -> registers; issued a tile ahead so that the latency hides behind the decode
__device__ __forceinline__ void k_units_load(KUnit &u, const kvc_qmeta_dev &m, long long tok0, long long T,
                                             long long b, long long h, int tid) {
    const int lane = tid & 31, sub = (tid >> 5) & 3;
    const long long t = tok0 + sub * 64;
    u.sc = make_uint2(0x3c003c00u, 0x3c003c00u); u.mi = make_uint2(0u, 0u);          // 1.0, 0
    if (m.sc != 0 && t < T) {                              // channel units lie side by side (sc == 1, checked by the host)
        const long long un = kvc_tok_unit(t, m.tok_div) * m.sj + b * m.sb + h * m.sh + lane * 4;
        u.sc = *reinterpret_cast<const uint2 *>(reinterpret_cast<const unsigned short *>(m.scale) + un);
        if (m.min_bytes == 1) u.mi.x = *reinterpret_cast<const uint32_t *>(reinterpret_cast<const int8_t *>(m.min_int) + un);
        else u.mi = *reinterpret_cast<const uint2 *>(reinterpret_cast<const int16_t *>(m.min_int) + un);
    }
}

template <int G>
__device__ __forceinline__ void k_weights_build(uint32_t *w, float *step, float *zp, const float *qf, const KUnit &u,
                                                bool channel_units, int min_bytes, long long tok0, long long T, int tid) {
    const int lane = tid & 31, wp = tid >> 5, sub = wp & 3;
    constexpr int GH = G >= 2 ? G / 2 : 1;
    if (G == 1 && wp >= 4) return;
    const bool live = tok0 + sub * 64 < T;
#pragma unroll
    for (int gi = 0; gi < GH; gi++) {
        const int g = G == 1 ? 0 : (wp >> 2) * GH + gi;
        float wv[4], z = 0.f;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float q = live ? qf[g * 128 + lane * 4 + i] : 0.f;
            const float sc = kvc_scale_value(ku_scale(u, i));
            wv[i] = q * sc;
            z = fmaf((float)ku_min(u, i, min_bytes) * sc, q, z);
        }
        float mx = fmaxf(fmaxf(fabsf(wv[0]), fabsf(wv[1])), fmaxf(fabsf(wv[2]), fabsf(wv[3])));
        mx = kvc_warp_max(mx);
        z = channel_units ? kvc_warp_sum(z) : 0.f;
        const float st = fix_step(mx), inv = st > 0.f ? 1.0f / st : 0.f;
        int q4[7];
#pragma unroll
        for (int i = 0; i < 4; i++) q4[i] = __float2int_rn(wv[i] * inv);
        uint32_t *row = w + (size_t)sub * 2 * WROW * G;
#pragma unroll
        for (int i = 0; i < 3; i++) {                           // the next lane's first three values
            int nv = __shfl_down_sync(0xffffffffu, q4[i], 1);
            q4[4 + i] = lane == 31 ? 0 : nv;
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {                           // layout: w_hi / w_lo
            const uint2 r = pack4(q4[i], q4[i + 1], q4[i + 2], q4[i + 3]);
            row[w_hi<G>(lane * 4 + i, g)] = r.x; row[w_lo<G>(lane * 4 + i, g)] = r.y;
        }
        if (lane < WROW - 128) { row[w_hi<G>(128 + lane, g)] = 0u; row[w_lo<G>(128 + lane, g)] = 0u; }
        if (lane == 0) { step[sub * G + g] = st; zp[sub * G + g] = z; }
    }
}

// The same in columns of bytes, for one block and the heads part * G/2 .. + G/2 - 1: w, step and zp are the block's, q the query heads [G][128],
// times the scaling; lane = 4 consecutive channels = one word.
template <int G>
__device__ __forceinline__ void k_weights_rows(uint32_t *w, float *step, float *zp, const float *q, const KUnit &u, bool channel_units, int min_bytes,
                                               int part, int lane) {
    constexpr int GP = G / 2;
    float sc[4], mz[4];
#pragma unroll
    for (int i = 0; i < 4; i++) { sc[i] = kvc_scale_value(ku_scale(u, i)); mz[i] = (float)ku_min(u, i, min_bytes) * sc[i]; }
    float z[GP];
#pragma unroll
    for (int gi = 0; gi < GP; gi++) {
        const int g = part * GP + gi;
        const float4 x = *reinterpret_cast<const float4 *>(q + g * 128 + lane * 4);
        const float w0 = x.x * sc[0], w1 = x.y * sc[1], w2 = x.z * sc[2], w3 = x.w * sc[3];
        z[gi] = fmaf(mz[0], x.x, fmaf(mz[1], x.y, fmaf(mz[2], x.z, mz[3] * x.w)));
        // The largest value of either sign (floats without a sign order as integers do).  The larger one takes the negative end of the range,
        // which reaches 32767; the positive end reaches 32639.
        const float up = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(fmaxf(fmaxf(w0, w1), fmaxf(w2, w3)), 0.f)) & 0x7fffffffu));
        const float down = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(fminf(fminf(fminf(w0, w1), fminf(w2, w3)), 0.f)) & 0x7fffffffu));
        const float big = fmaxf(up, down), st = fmaxf(big * (1.0f / FIX_DOWN), fminf(up, down) * (1.0f / FIX_UP));
        const float inv = big > 1e-30f ? rcp_fast(st) : 0.f;
        const uint2 r = pack_fix(w0, w1, w2, w3, up > down ? -inv : inv);
        w[2 * g * COL_WORDS + lane] = r.x; w[(2 * g + 1) * COL_WORDS + lane] = r.y;
        if (lane == 0) step[g] = up > down ? -st : st;
    }
    if (!channel_units) { if (lane < GP) zp[part * GP + lane] = 0.f; return; }
#pragma unroll
    for (int gi = 0; gi < GP; gi += 2) {                    // two heads' sums in one go: one to either half of the warp
        float a = z[gi];
        if (GP > 1) {
            const float z1 = z[(gi + 1) % GP];
            const float give = lane < 16 ? z1 : a;
            a = (lane < 16 ? a : z1) + __shfl_xor_sync(0xffffffffu, give, 16);
        } else a += __shfl_xor_sync(0xffffffffu, a, 16);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        if ((lane & 15) == 0 && (GP > 1 || lane == 0)) zp[part * GP + gi + (lane >> 4)] = a;
    }
}

template <int G>
__device__ __forceinline__ void k_weights(uint32_t *w, float *step, float *zp, const float *qf, const kvc_qmeta_dev &m,
                                          long long tok0, long long T, long long b, long long h, int tid) {
    KUnit u;
    k_units_load(u, m, tok0, T, b, h, tid);
    k_weights_build<G>(w, step, zp, qf, u, m.sc != 0, m.min_bytes, tok0, T, tid);
}

template <int G>
__device__ __forceinline__ void load_q(float *qf, float *qsum, const __half *q, long long b, long long Hq,
                                       long long hq0, float scaling, int tid) {
    for (int i = tid; i < G * 128; i += NTHR) {
        const int g = i >> 7, c = i & 127;
        qf[i] = __half2float(q[(b * Hq + hq0 + g) * 128 + c]) * scaling;
    }
    __syncthreads();
    if (tid < G * 32) {           // one warp per query head
        const int g = tid >> 5, lane = tid & 31;
        float s = qf[g * 128 + lane] + qf[g * 128 + lane + 32] + qf[g * 128 + lane + 64] + qf[g * 128 + lane + 96];
        s = kvc_warp_sum(s);
        if (lane == 0) qsum[g] = s;
    }
}

// scale and min_int of a token whose K units do not depend on the channel (loaded ahead of the decode)
__device__ __forceinline__ void k_token_unit(unsigned short &sc, int &mi, const kvc_qmeta_dev &m, long long t,
                                             long long b, long long h) {
    const long long u = kvc_tok_unit(t, m.tok_div) * m.sj + b * m.sb + h * m.sh;
    sc = kvc_load_scale_bits(m, u); mi = kvc_load_min(m, u);
}

// score of the thread's token from its integer dot products
template <int G>
__device__ __forceinline__ void k_finish(float (&s)[G], const int (&hi)[G], const int (&lo)[G], const float *step_sub,
                                         const float *zp_sub, const float *qsum, bool channel_units, float sc, float mi) {
#pragma unroll
    for (int g = 0; g < G; g++) {
        const float d = fix_value(step_sub[g], hi[g], lo[g]);
        s[g] = channel_units ? d + zp_sub[g] : sc * fmaf(mi, qsum[g], d);
    }
}

// ---- V weights --------------------------------------------------------------------------------------
// Called by all 256 threads (thread = token of the tile, grp = its 128-token group, tl = its index in
// the group) with wv[g] = p[g] * scale of the token.  Builds records ps[grp][tl][hi|lo][g], step[grp][g].
// `red` is scratch for 8*G floats, `q16` for 2*G*(128+4) int16.  Contains three block barriers.
template <int G>
__device__ __forceinline__ void v_weights(uint32_t *ps, float *vstep, float *red, int16_t *q16, const float (&wv)[G],
                                          int tid) {
    const int lane = tid & 31, warp = tid >> 5, grp = tid >> 7, tl = tid & 127;
#pragma unroll
    for (int g = 0; g < G; g++) { float mx = kvc_warp_max(fabsf(wv[g])); if (lane == 0) red[warp * G + g] = mx; }
    if (tl < 4) for (int g = 0; g < G; g++) q16[(grp * G + g) * 132 + 128 + tl] = 0;
    __syncthreads();
#pragma unroll
    for (int g = 0; g < G; g++) {
        const float mx = fmaxf(fmaxf(red[(grp * 4 + 0) * G + g], red[(grp * 4 + 1) * G + g]),
                               fmaxf(red[(grp * 4 + 2) * G + g], red[(grp * 4 + 3) * G + g]));
        const float st = fix_step(mx);
        q16[(grp * G + g) * 132 + tl] = (int16_t)fix_quant(wv[g], st);
        if (tl == 0) vstep[grp * G + g] = st;
    }
    __syncthreads();
#pragma unroll
    for (int g = 0; g < G; g++) {
        const int16_t *qq = q16 + (grp * G + g) * 132 + tl;
        uint32_t *row = ps + (size_t)grp * 2 * WROW * G;    // layout: w_hi / w_lo
        const uint2 r = pack4(qq[0], qq[1], qq[2], qq[3]);
        row[w_hi<G>(tl, g)] = r.x; row[w_lo<G>(tl, g)] = r.y;
        if (tl < WROW - 128) { row[w_hi<G>(128 + tl, g)] = 0u; row[w_lo<G>(128 + tl, g)] = 0u; }
    }
    __syncthreads();
}

// ---- fused K: raw scores ------------------------------------------------------------------------
// Both unfused kernels: the structure, four staging slots sized by the stream's largest block, SLOT_PAD bytes that a
// corrupt stream's overrun may read.  (Slots for the largest block of the format let three CTAs share an SM; with the
// stream's own, six do.)
template <class S> size_t unfused_smem(const CacheDev &c) { return sizeof(S) + 4 * (size_t)slot_bytes_of(c.max_block) + SLOT_PAD; }
template <int G>
struct alignas(32) QkSmem {
    KvcBookSmem book;
    alignas(32) uint32_t w[4 * 2 * WROW * G];
    float step[4 * G];
    float zp[4 * G];
    float qf[G * 128];
    float qsum[G];
    uint32_t lead[4], nb[4];
    int ok[4];
};

template <int G>
__global__ void __launch_bounds__(NTHR) fused_qk_kernel(CacheDev kc, long long T, long long B, long long Hkv, long long Hq,
                                                        long long g0, const __half *__restrict__ q, void *__restrict__ out,
                                                        int out_f32, int *__restrict__ status) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    QkSmem<G> &sm = *reinterpret_cast<QkSmem<G> *>(smem_raw);
    uint8_t *const slot = smem_raw + sizeof(QkSmem<G>) + (threadIdx.x >> 6) * slot_bytes_of(kc.max_block);
    const int tid = threadIdx.x, sub = tid >> 6, v = tid & 63;
    const long long cols = B * Hkv, col = blockIdx.y, b = col / Hkv, h = col % Hkv;
    const long long Gt = Hq / Hkv, hq0 = h * Gt + g0;
    const long long tok0 = (long long)blockIdx.x * 256, t = tok0 + tid;
    kvc_load_book(sm.book, kc.book, tid, NTHR);
    const bool esc = book_has_long_codes(kc.book);
    load_q<G>(sm.qf, sm.qsum, q, b, Hq, hq0, 1.0f, tid);
    const long long blk = (tok0 / 64 + sub) * cols + col;
    const bool active = t < T;
    if (active) { uint32_t ld, nb; bool ok = stage(kc, blk, slot, &ld, &nb, v); if (v == 0) { sm.lead[sub] = ld; sm.nb[sub] = nb; sm.ok[sub] = ok; } }
    __syncthreads();
    k_weights<G>(sm.w, sm.step, sm.zp, sm.qf, kc.q, tok0, T, b, h, tid);
    __syncthreads();
    if (!active) return;
    unsigned short ksc = 0x3c00; int kmi = 0;
    if (kc.q.sc == 0) k_token_unit(ksc, kmi, kc.q, t, b, h);
    int hi[G], lo[G];
#pragma unroll
    for (int g = 0; g < G; g++) { hi[g] = 0; lo[g] = 0; }
    const uint32_t start = vec_start(kc.thread_info, blk, v);
    bool ok = sm.ok[sub] && start < sm.nb[sub];                // a vector begins inside its block
    if (ok) ok = decode_dot<G>(slot, sm.lead[sub] + start, sm.book, esc, sm.w + sub * 2 * WROW * G, hi, lo);
    if (!ok) atomicOr(status, KVC_FLAG_BAD_STREAM);
    float s[G];
    k_finish<G>(s, hi, lo, sm.step + sub * G, sm.zp + sub * G, sm.qsum, kc.q.sc != 0, kvc_scale_value(ksc), (float)kmi);
#pragma unroll
    for (int g = 0; g < G; g++) {
        const long long o = (b * Hq + hq0 + g) * T + t;
        if (out_f32) reinterpret_cast<float *>(out)[o] = s[g];
        else reinterpret_cast<__half *>(out)[o] = __float2half_rn(s[g]);
    }
}

// ---- fused V: per-group partial outputs ----------------------------------------------------------
template <int G>
struct alignas(32) PvSmem {
    KvcBookSmem book;
    alignas(32) uint32_t ps[2 * 2 * WROW * G];
    float vstep[2 * G];
    float zpv[2 * G];
    float red[2][8 * G];
    int16_t q16[2 * G * 132];
    uint32_t lead[4], nb[4];
    int ok[4];
};

template <int G>
__global__ void __launch_bounds__(NTHR, 6) fused_pv_kernel(CacheDev vc, long long T, long long B, long long Hkv, long long Hq,
                                                        long long g0, const __half *__restrict__ P, __half *__restrict__ out,
                                                        int *__restrict__ status) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    PvSmem<G> &sm = *reinterpret_cast<PvSmem<G> *>(smem_raw);
    uint8_t *const slot = smem_raw + sizeof(PvSmem<G>) + (threadIdx.x >> 6) * slot_bytes_of(vc.max_block);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, sub = tid >> 6, v = tid & 63;
    const int grp = tid >> 7, ch = tid & 127;
    const long long cols = B * Hkv, col = blockIdx.y, b = col / Hkv, h = col % Hkv;
    const long long Gt = Hq / Hkv, hq0 = h * Gt + g0;
    const long long tok0 = (long long)blockIdx.x * 256, t = tok0 + tid;
    const kvc_qmeta_dev &m = vc.q;
    kvc_load_book(sm.book, vc.book, tid, NTHR);
    const bool esc = book_has_long_codes(vc.book);
    const long long gI = tok0 / 128 + grp;
    const long long blk = gI * (cols * 2) + col * 2 + (ch >> 6);
    const bool active = gI * 128 < T;
    if (active) { uint32_t ld, nb; bool ok = stage(vc, blk, slot, &ld, &nb, v); if (v == 0) { sm.lead[sub] = ld; sm.nb[sub] = nb; sm.ok[sub] = ok; } }
    float wv[G];
    {
        float sc = 0.f, mi = 0.f;
        if (t < T) {
            const long long u = kvc_tok_unit(t, m.tok_div) * m.sj + b * m.sb + h * m.sh;
            sc = __half2float(m.scale[u]); mi = (float)kvc_load_min(m, u);
        }
#pragma unroll
        for (int g = 0; g < G; g++) {
            const float p = t < T ? __half2float(P[(b * Hq + hq0 + g) * T + t]) : 0.f;
            wv[g] = p * sc;
            const float z = kvc_warp_sum(wv[g] * mi);
            if (lane == 0) sm.red[1][warp * G + g] = z;
        }
    }
    v_weights<G>(sm.ps, sm.vstep, sm.red[0], sm.q16, wv, tid);
    if (!active) return;
    int hi[G], lo[G];
#pragma unroll
    for (int g = 0; g < G; g++) { hi[g] = 0; lo[g] = 0; }
    const uint32_t start = vec_start(vc.thread_info, blk, v);
    bool ok = sm.ok[sub] && start < sm.nb[sub];
    if (ok) ok = decode_dot<G>(slot, sm.lead[sub] + start, sm.book, esc, sm.ps + grp * 2 * WROW * G, hi, lo);
    if (!ok) atomicOr(status, KVC_FLAG_BAD_STREAM);
#pragma unroll
    for (int g = 0; g < G; g++) {
        const float z = sm.red[1][(grp * 4 + 0) * G + g] + sm.red[1][(grp * 4 + 1) * G + g] +
                        sm.red[1][(grp * 4 + 2) * G + g] + sm.red[1][(grp * 4 + 3) * G + g];
        out[((gI * B + b) * Hq + hq0 + g) * 128 + ch] = __float2half_rn(fix_value(sm.vstep[grp * G + g], hi[g], lo[g]) + z);
    }
}

// ---- one-pass decode attention -------------------------------------------------------------------
struct AttnParams {
    CacheDev k, v;
    long long T, B, Hkv, Hq, Tr;
    long long g0;                 // first query head of this launch (of each KV head)
    int nh;                       // and how many, 1 .. G
    const __half *q, *ktail, *vtail;
    __half *out;
    float scaling;
    int n_tiles;                  // steps of 128 tokens per column
    // every column is cut into `long_runs` runs of `tiles_per_split` steps followed by `splits - long_runs`
    // runs of `short_tiles` steps; the items of the long runs of all columns come first, the short ones last
    int splits, tiles_per_split, long_runs, short_tiles;
    long long work;               // columns * splits items
    uint32_t slotK_bytes, slotV_bytes;   // capacity of one staging slot (multiple of 16)
    float *ws_part;               // [B*Hq][splits][ROWS_PART_FLOATS]
    int *sched;                   // {items handed out, workers finished}, or null: static shares
    int *status;
    int workers;                  // per CTA
    int brief;                    // BRIEF_STEPS steps per worker at most: vectors are decoded whole
    int spare;                    // there is room for a table of V's single symbols beside that of pairs
    int team;                     // without partial results: this many workers of a CTA share a column's steps and add up in shared memory (0: each its own columns)
    int partial;                  // items leave partial results for the merge kernel (several runs per column, or a tail that the merge kernel adds)
    int early;                    // one head: the merge kernel is let go when a worker of every CTA has no further item, else when one has ended
    int wait_limit;               // tries of a staging wait before it gives up (KVC_FLAG_WAIT_TIMEOUT)
    int starve;                   // tests of the bounded waits only: announce bytes that are never copied
};

// ---- grouped queries: the same attention with workers of 128 threads --------------------------------
// A CTA is one resident per SM, with one copy of the two decode tables and up to five (eight heads: four) workers.
// A worker is four warps with slots, rows, weights and barriers of its own; it draws items and walks them in steps of 128
// tokens (two K blocks, the two V blocks of a column), with three barriers per step: K's weights are in, the largest score is known, V's
// weights are in.  Threads beyond the workers that a launch needs help to load the tables.
constexpr int ROWS_PART_FLOATS = 130;        // a partial result: m, l, acc[128]
static_assert(2 * ROWS_PART_FLOATS <= ATTN_PART_FLOATS, "a workspace for n runs of 256-token tiles holds 2 n partial results");
template <int G> __host__ __device__ constexpr int rows_workers() { return G == 8 ? 4 : 5; }
// Bytes of 128 symbols from which a vector has too many windows of one code for pairs: 5 bits a symbol.  (16 x 16384 tokens, 8 x 4 heads, one V channel of every head
// six times the others, units of V per token at rel 0.05, and per token and head at 0.1: by pairs, with what fell behind again symbol by symbol, 517 and 523 us, at the
// lane's own pace 439 and 456, from the spare table 343 and 380; from 88 bytes on 343 and 398, from 96 on 366 and 404.  A book that goes by pairs has 4.1 bits a symbol at most, 66
// bytes a vector on average.)
constexpr uint32_t LONG_VECTOR = 80;
constexpr int ROWS_PLANNED = 5;              // workers per SM that the plan of a grouped launch counts

template <int G>
struct alignas(32) RowsWorker {
    uint32_t w[3 * vec_words(G)];            // weight words: K of the step's two blocks, V; scratch of the tail and of a team's sums
    float q[G * 128];                        // the query, times the scaling
    float vsc[128], vz[128], vlg[128];       // of the step's tokens: V's scale, scale * min_int, log of the scale
    float red[G][4];                         // per-warp partials of a head
    float kstep[2 * G], zp[2 * G], qsum[G];
    uint64_t bar[2];                         // K and V staging barriers
    uint32_t leadK[4], leadV[4], nbK[4], nbV[4];   // of the two staged blocks (stage_bulk writes four entries)
    int okK[4], okV[4];
    int next_j, dead;
};
struct alignas(32) OneTables { uint32_t lutK[KVC_LUT_SIZE], lutV[KVC_LUT_SIZE]; };       // (the one-head kernel reads its trees from global memory)
struct RowsTables : OneTables { uint32_t tree[2][512]; uint8_t len[512]; };              // the trees are for codes beyond the window

// shared memory of a CTA: tables, workers, slots (two of K and two of V each), rows; a corrupt stream's overrun ends in the rows
template <int G> size_t rows_smem(const AttnParams &p, int workers) {
    return sizeof(RowsTables) + workers * (sizeof(RowsWorker<G>) + 2 * (size_t)(p.slotK_bytes + p.slotV_bytes) + 128 * (p.brief ? WHOLE_ROW_BYTES : ROW_BYTES)) +
           (p.spare ? 4 * KVC_LUT_SIZE : 0);
}

template <int G> int rows_fit(const AttnParams &p) {         // workers that an SM holds
    int workers = rows_workers<G>();
    while (workers > 1 && rows_smem<G>(p, workers) > MAX_CTA_SHARED) workers--;
    return workers;
}
int one_fit(const AttnParams &p);
int rows_fit(const AttnParams &p, int heads) { return heads == 1 ? one_fit(p) : heads > 4 ? rows_fit<8>(p) : (heads > 2 ? rows_fit<4>(p) : rows_fit<2>(p)); }

// Equal items for `most` takers per SM: in how many rounds they go, and the takers that this many rounds need: those of a
// fuller SM would run slower and the last round leave more of them idle.  (One head, seven workers at first, device time: 320 columns
// of 6144 tokens in 4 runs 254 us, now 229 (three CTAs of 256 threads, the kernel before the workers: 250); 192 of 4096 in 6 runs 127 and 107; 36 of
// 4096, the library's plan, 36 and 27; 800 columns of 128 tokens, 4 heads, 34 and 28.)
struct Spread { long long rounds, per_sm; };
Spread spread(long long items, long long most, long long sms) {
    const long long rounds = (items + most * sms - 1) / (most * sms);
    return {rounds, (items + rounds * sms - 1) / (rounds * sms)};
}

// How many of an SM's workers share a column when every column's output is written directly (no workspace, or a single run
// without a tail): without company a worker would take all of a column's `units` (steps and passes of the tail) in turn
// while most of the device is idle.  A unit takes about 6 + a parts of time with `a` workers at work on the SM (2 heads: 7.1 us
// alone, 11.9 us with five), a team's sums and its next column another 3.5 (fitted to steps of 9.2 and 14.4 us: over 1 to 700 columns of 2 to 19 units the
// choice was within 1 % of the best size on average, and nowhere behind a worker per column).  2 heads per column, no workspace, a worker per column
// against teams: 8 columns of 1024 tokens 53.3 and 26.6 us, 64 of 8192 457 and 148 us, 256 of 256 (two teams of two on an SM) 22.1 and
// 16.8 us; more columns than workers, where a worker per column goes in two rounds, the second nearly empty: 1280 of 1024 tokens,
// one head, 236 and 165 us.
int rows_team(long long cols, long long units, int workers, int sms) {       // (0: each its own columns)
    int best = 0;
    long long least = 0;
    for (int size = 1; size <= workers && size <= units; size++) {
        const Spread s = spread(cols, workers / size, sms);
        const long long teams = s.per_sm, cost = s.rounds * (2 * ((units + size - 1) / size) * (6 + teams * size) + (size > 1 ? 7 : 0));
        if (size == 1 || cost < least) { least = cost; best = size > 1 ? size : 0; }
    }
    return best;
}

// TEAM: see rows_team (a kernel of its own: a branch on it costs the other one 0.8 % through registers alone).
template <int G, bool BULK, bool TEAM>
__global__ void __launch_bounds__(128 * rows_workers<G>(), 1) attn_rows_kernel(AttnParams p) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    RowsTables &tab = *reinterpret_cast<RowsTables *>(smem_raw);
    constexpr int HL = G == 8 ? 2 : 1;                     // heads per lane
    constexpr int VW = vec_words(G);
    const int workers = p.workers, wk = threadIdx.x >> 7;      // (threads beyond the workers help to load the tables)
    const int tid = threadIdx.x & 127, lane = tid & 31, warp = tid >> 5, sub = warp >> 1;
    // The lane decodes vector `vec` of the step, and holds the results of the vectors 4 r .. 4 r + 3 of its warp (tokens in the K phase,
    // channels in the V phase) for the heads q4 % G and, with eight, q4 + 4.
    const int vec = warp * 32 + vec_of_lane(lane), v = vec & 63;
    const int r4 = lane & ~3, q4 = lane & 3, hd = q4 % G;
    const bool own = q4 < G;                               // with two heads the other lanes hold copies
    uint8_t *const wbase = smem_raw + sizeof(RowsTables), *const sbase = wbase + workers * sizeof(RowsWorker<G>);
    RowsWorker<G> &sm = reinterpret_cast<RowsWorker<G> *>(wbase)[wk];
    uint8_t *const slotsK = sbase + wk * 2 * (p.slotK_bytes + p.slotV_bytes), *const slotsV = slotsK + 2 * p.slotK_bytes;
    const uint32_t rows_s = kvc_smem_addr(sbase + workers * 2 * (p.slotK_bytes + p.slotV_bytes)) + (wk * 4 + warp) * 32 * (p.brief ? WHOLE_ROW_BYTES : ROW_BYTES);
    uint32_t *const spare = reinterpret_cast<uint32_t *>(sbase + workers * (2 * (p.slotK_bytes + p.slotV_bytes) + 128 * ROW_BYTES));      // (never with brief)
    auto sync = [&]() { asm volatile("bar.sync %0, 128;" :: "r"(wk + 1) : "memory"); };     // the worker's threads
    auto release = []() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); };
    // launched with programmatic stream serialisation: this kernel's own set-up -- the tables, the first blocks, the first step's metadata: cache
    // data that no kernel of a decode step writes -- runs before griddepcontrol.wait, possibly while the kernel ahead of it in the
    // stream (the merge of the layer before, which lets its dependents start early) still runs.  What that kernel or the one before it may
    // write (the query, the scheduling counters, the workspace, the output, the status word) is touched after the wait.  This kernel's own
    // dependent, the merge kernel, is let go when a worker of every CTA has no further item, and never before the wait, as it reads the query and the tail's rows
    // right away: it is set up, and has added up the tail, by the time that the last worker ends.  (It started 2.1 us after the last CTA's end and took 4 to 6 us for
    // a tail.  Launch pair, device time, let go by the end of the CTAs and now: 12 columns of 2816 tokens and 165 rows, 6 heads, 22.3 and 17.1 us; 16 of 896 and 150, 4
    // heads, 19.6 and 14.2; 32 of 1024, one head, no tail, 15.3 and 13.6; 256 of 4096 and 128 rows, one head, 128.8 and 123.2; 128 columns of 4096 and 128, 4 heads, 99.3 and
    // 94.9; 16 of 16384, 49.1 and 45.9; 8 of 16384 30.9 and 31.1, of 32768 47.5 and 47.8.  Let go by a worker's end 126.2 where 123.2 stand, 18.7 where let go by its last item gives 17.1; at
    // the kernel's top, whatever the items, 49.2 us where 47.8 stand.)
    const int B = (int)p.B, Hkv = (int)p.Hkv, Hq = (int)p.Hq;
    const int cols = B * Hkv, Gt = Hq / Hkv;
    const kvc_qmeta_dev &km = p.k.q, &vm = p.v.q;
    int flags = 0;

    struct Item { int col, t_lo, t_hi, part; };            // steps t_lo .. t_hi - 1 of a column; part: the run's index
    const bool draw = !TEAM && p.sched != nullptr;
    const int P = (int)gridDim.x * (TEAM ? workers / p.team : workers);
    const int me = TEAM ? wk / p.team * (int)gridDim.x + (int)blockIdx.x : (int)blockIdx.x * workers + wk;
    const int w_hi = draw ? (int)p.work : (int)(p.work * (me + 1) / P);
    auto item_of = [&](int j, Item &it) -> bool {
        if (j >= w_hi) return false;
        const int n_long = cols * p.long_runs;
        if constexpr (TEAM) {                              // the worker's share of column j: the same for every column
            const int tk = wk % p.team;
            it.col = j; it.part = 0; it.t_lo = (int)((long long)p.n_tiles * tk / p.team); it.t_hi = (int)((long long)p.n_tiles * (tk + 1) / p.team);
        } else if (j < n_long) {
            const int r = j % p.long_runs;
            it.col = j / p.long_runs; it.part = r; it.t_lo = r * p.tiles_per_split; it.t_hi = min(p.n_tiles, it.t_lo + p.tiles_per_split);
        } else {
            const int n_short = p.splits - p.long_runs, r = (j - n_long) % n_short;
            it.col = (j - n_long) / n_short; it.part = p.long_runs + r;
            it.t_lo = p.long_runs * p.tiles_per_split + r * p.short_tiles; it.t_hi = min(p.n_tiles, it.t_lo + p.short_tiles);
        }
        return true;
    };
    auto blkK_of = [&](int col, int t, int l) { return ((long long)t * 2 + l) * cols + col; };
    auto blkV_of = [&](int col, int t, int l) { return (long long)t * (cols * 2) + (long long)col * 2 + l; };

    Item it, nit;
    // The first item is fixed by the worker's index; with a counter, the next one is drawn when an item begins and looked at in its last step, when
    // that step's blocks are asked for.  (Drawn an item earlier, a worker held two when the counter ran out.)
    int j_n1 = draw ? me : (int)(p.work * me / P);
    bool have = wk < workers && item_of(j_n1, it), have_next = false;
    if (!draw) have_next = have && item_of(++j_n1, nit);
    const bool more = draw && p.work > P;                  // not all of the items are fixed
    int drawn = 0;                                         // thread 0: the counter's answer
    const bool any = have && it.t_lo < it.t_hi;

    // the two blocks of a step, by the lanes 0 and 1 of the worker's first warp
    auto stage_K = [&](bool on, int col, int t) { stage_bulk(p.k, on && lane < 2, blkK_of(col, t, lane & 1), slotsK + (lane & 1) * p.slotK_bytes, sm.leadK, sm.okK, sm.nbK, &sm.bar[0], lane, p.starve != 0); };
    auto stage_V = [&](bool on, int col, int t) { stage_bulk(p.v, on && lane < 2, blkV_of(col, t, lane & 1), slotsV + (lane & 1) * p.slotV_bytes, sm.leadV, sm.okV, sm.nbV, &sm.bar[1], lane, p.starve != 0); };
    if (BULK && wk < workers) {
        if (tid == 0) { kvc_mbar_init(&sm.bar[0], 1); kvc_mbar_init(&sm.bar[1], 1); kvc_mbar_fence_init(); sm.dead = 0; }
        sync();
        if (warp == 0 && any) { stage_K(true, it.col, it.t_lo); stage_V(true, it.col, it.t_lo); }
    }
    const KvcWay wayK = kvc_book_way(p.k.book, p.brief != 0), wayV = kvc_book_way(p.v.book, p.brief != 0);
    const bool spare_in = p.spare && wayV.way == KVC_PAIRS;
    if (p.brief) {
        kvc_load_luts(tab.lutK, tab.lutV, p.k.book, p.v.book, threadIdx.x, blockDim.x);
    } else kvc_load_ways(tab.lutK, tab.lutV, spare_in ? spare : nullptr, p.k.book, p.v.book, wayK.way == KVC_PAIRS, wayV.way == KVC_PAIRS, tab.len, threadIdx.x, blockDim.x);
    if (wayK.esc) kvc_load_tree(tab.tree[0], p.k.book, threadIdx.x, blockDim.x);
    if (wayV.esc) kvc_load_tree(tab.tree[1], p.v.book, threadIdx.x, blockDim.x);
    const uint32_t lutK_s = kvc_smem_addr(tab.lutK), lutV_s = kvc_smem_addr(tab.lutV), tree_s = kvc_smem_addr(tab.tree), loneV_s = spare_in ? kvc_smem_addr(spare) : lutV_s;

    struct StepMeta { unsigned short startK, startV, vsc, ksc; int vmi, kmi; KUnit ku; };   // as loaded: no arithmetic waits on them here
    auto load_meta = [&](bool on, int b, int h, int col, int step, StepMeta &m) {
        m.startK = m.startV = 0; m.vsc = 0; m.vmi = m.kmi = 0; m.ksc = 0x3c00;
        m.ku.sc = make_uint2(0x3c003c00u, 0x3c003c00u); m.ku.mi = make_uint2(0u, 0u);          // 1.0, 0
        if (!on) return;
        // (token and block numbers fit 32 bits: the host's check, and the tables' size)
        m.startK = vec_start_bits32(p.k.thread_info, (uint32_t)(step * 2 + sub) * (uint32_t)cols + (uint32_t)col, v);
        m.startV = vec_start_bits32(p.v.thread_info, ((uint32_t)step * (uint32_t)cols + (uint32_t)col) * 2u + (uint32_t)sub, v);
        const uint32_t t = (uint32_t)(step * 128 + vec);
        const long long u = unit_of(vm, vm.tok_div == 1 ? t : t / (uint32_t)vm.tok_div, b, h);
        m.vsc = kvc_load_scale_bits(vm, u); m.vmi = kvc_load_min(vm, u);
        if (km.sc == 0) {
            const long long uk = unit_of(km, km.tok_div == 1 ? t : t / (uint32_t)km.tok_div, b, h);
            m.ksc = kvc_load_scale_bits(km, uk); m.kmi = kvc_load_min(km, uk);
        } else {                                           // of the block whose weights the warp builds (warp & 1), 4 channels per lane
            const uint32_t blk = (uint32_t)(step * 2 + (warp & 1));
            const long long un = unit_of(km, km.tok_div == 64 ? blk : blk * 64u / (uint32_t)km.tok_div, b, h) + lane * 4;
            m.ku.sc = *reinterpret_cast<const uint2 *>(reinterpret_cast<const unsigned short *>(km.scale) + un);
            if (km.min_bytes == 1) m.ku.mi.x = *reinterpret_cast<const uint32_t *>(reinterpret_cast<const int8_t *>(km.min_int) + un);
            else m.ku.mi = *reinterpret_cast<const uint2 *>(reinterpret_cast<const int16_t *>(km.min_int) + un);
        }
    };
    StepMeta cur;
    load_meta(any, have ? it.col / Hkv : 0, have ? it.col % Hkv : 0, have ? it.col : 0, have ? it.t_lo : 0, cur);
    unsigned short qn[G];                                  // the query of an item is fetched while the item before it runs
    auto q_fetch = [&](int col_) {
        const long long row0 = (long long)(col_ / Hkv) * Hq + (long long)(col_ % Hkv) * Gt + p.g0;
#pragma unroll
        for (int g = 0; g < G; g++) qn[g] = g < p.nh ? reinterpret_cast<const unsigned short *>(p.q)[(row0 + g) * 128 + tid] : (unsigned short)0;
    };
    __syncthreads();                                       // the tables are in; from here on the workers go their own ways
    if (wk >= workers) return;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (have) q_fetch(it.col);

    // over a warp's vectors: the lane's four, then the eight lanes with the same heads
    auto warp_max = [&](float x) { x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 4)); x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 8)); return fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 16)); };
    auto warp_sum = [&](float x) { x += __shfl_xor_sync(0xffffffffu, x, 4); x += __shfl_xor_sync(0xffffffffu, x, 8); return x + __shfl_xor_sync(0xffffffffu, x, 16); };
    auto red_max = [&](int g) { const float4 x = *reinterpret_cast<const float4 *>(sm.red[g]); return fmaxf(fmaxf(x.x, x.y), fmaxf(x.z, x.w)); };
    auto red_sum = [&](int g) { const float4 x = *reinterpret_cast<const float4 *>(sm.red[g]); return (x.x + x.y) + (x.z + x.w); };

    uint32_t par = 0;                                      // bit 0 / bit 1: parity of the staging phase the K / V barrier is waited for next; bit 2: the item's V from the spare table
    bool v_staged = any, v_landed = true;                  // V blocks of the step to come are on their way already; the last wait for them ended well
    while (have) {
    const int col = it.col, b = col / Hkv, h = col % Hkv;
    if (!more && !have_next) release();
    if (more && tid == 0) drawn = atomicAdd(&p.sched[0], 1);
#pragma unroll
    for (int g = 0; g < G; g++) sm.q[g * 128 + tid] = kvc_scale_value(qn[g]) * p.scaling;
    sync();
    if (km.sc == 0) for (int g = warp; g < G; g += 4) {    // sum of each query head's 128 (scaled) values
        float a = 0.f;
#pragma unroll
        for (int k = 0; k < 4; k++) a += sm.q[g * 128 + k * 32 + lane];
        a = kvc_warp_sum(a);
        if (lane == 0) sm.qsum[g] = a;
    }
    // A channel far beyond the others of its tokens has nothing but long codes, in every step of the column.  A warp with a vector of more than LONG_VECTOR
    // bytes in the first step (up to where the next one begins; that of the warp's last is not known) takes the item's V one symbol per lookup, from
    // the spare table.
    if (spare_in) {
        const uint32_t at = cur.startV >> 3, bytes = __shfl_sync(0xffffffffu, at, lane < 24 ? lane + 8 : (lane + 1) & 7) - at;
        par = __any_sync(0xffffffffu, bytes > LONG_VECTOR && lane != 31) ? par | 4u : par & 3u;
    }
    // acc: the lane's four channels.  l, z: the sums of the weights and of weight * scale * min_int over the lane's own tokens, added up
    // over the lanes at the item's end.  All relative to e^m.
    float m_run[HL], l_run[HL], z_run[HL], acc[4][HL];
#pragma unroll
    for (int j = 0; j < HL; j++) {
        m_run[j] = -CUDART_INF_F; l_run[j] = z_run[j] = 0.f;
#pragma unroll
        for (int i = 0; i < 4; i++) acc[i][j] = 0.f;
    }

    for (int step = it.t_lo; step < it.t_hi; step++) {
        if (!BULK) {
            if (step != it.t_lo) sync();                   // every thread is done with the V slots
            const int sb = tid >> 6, sv = tid & 63;
            uint32_t ld, nb;
            bool ok = stage(p.k, blkK_of(col, step, sb), slotsK + sb * p.slotK_bytes, &ld, &nb, sv);
            if (sv == 0) { sm.leadK[sb] = ld; sm.nbK[sb] = nb; sm.okK[sb] = ok; }
            ok = stage(p.v, blkV_of(col, step, sb), slotsV + sb * p.slotV_bytes, &ld, &nb, sv);
            if (sv == 0) { sm.leadV[sb] = ld; sm.nbV[sb] = nb; sm.okV[sb] = ok; }
        }
        k_weights_rows<G>(sm.w + (warp & 1) * VW, sm.kstep + (warp & 1) * G, sm.zp + (warp & 1) * G, sm.q, cur.ku, km.sc != 0, km.min_bytes, warp >> 1, lane);
        {
            const float sc = kvc_scale_value(cur.vsc);     // of the token `vec`; read by lanes of the same warp
            sm.vsc[vec] = sc; sm.vz[vec] = sc * (float)cur.vmi; // (at least fp16's smallest; a negative scale's weights take the shorter end of the fixed-point range)
            sm.vlg[vec] = log2_fast(fmaxf(fabsf(sc), 5.9604645e-8f)) * LN2 + (sc < 0.f ? 0.0077f : 0.f);      // (32880 * exp(-0.0077) < 32639)
        }
        bool k_landed = true;                              // (a wait that runs out: see attn_one_kernel)
        if (BULK) {
            k_landed = kvc_mbar_wait(&sm.bar[0], par & 1u, p.wait_limit);
            if (k_landed) par ^= 1u; else flags |= KVC_FLAG_WAIT_TIMEOUT;
        }
        sync();                                            // also: every thread is done with the V slots of the step before
        if (BULK && warp == 0 && !v_staged) {              // this step's V blocks land during its K phase
            if (__all_sync(0xffffffffu, v_landed)) stage_V(true, col, step);
            else if (lane == 0) sm.dead = 1;
        }
        // ---- K: scores of this step's tokens
        float s[4][HL];
        {
            int d[4][HL];
            const uint32_t start = cur.startK >> 3;
            bool ok = k_landed && sm.okK[sub] && start < sm.nbK[sub];              // a vector begins inside its block
            uint32_t lagged = 0;
            ok = rows_dot<G>(wayK, {kvc_smem_addr(slotsK + sub * p.slotK_bytes), ok ? sm.leadK[sub] + start : 1u, lutK_s, lutK_s, tree_s}, rows_s, kvc_smem_addr(sm.w + sub * VW), lane, d, lagged) && ok;
            if (!ok) flags |= KVC_FLAG_BAD_STREAM;
            const uint32_t unit = (uint32_t)cur.ksc | ((uint32_t)cur.kmi << 16);   // of the token `vec`
#pragma unroll
            for (int j = 0; j < HL; j++) {
                const float st = sm.kstep[sub * G + hd + 4 * j], z = sm.zp[sub * G + hd + 4 * j];
#pragma unroll
                for (int i = 0; i < 4; i++) s[i][j] = fmaf(st, (float)d[i][j], z);
            }
            if (km.sc == 0) {
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const uint32_t u = __shfl_sync(0xffffffffu, unit, (lane >> 2) + 8 * i);
                    const float sc = kvc_scale_value((unsigned short)u), mi = (float)((int)u >> 16);
#pragma unroll
                    for (int j = 0; j < HL; j++) s[i][j] = sc * fmaf(mi, sm.qsum[hd + 4 * j], s[i][j]);
                }
            }
        }
        // ---- online softmax over the step.  The reference of a step is the largest of weight * V scale over its tokens, i.e. of score + log of
        // the scale: the V weights are then at most 1, and their fixed-point step is known without another exchange.  (The sums are rounded up: rounded
        // to nearest, half an ulp of a score of 1e5 took the largest weight beyond 16 bits.)
        const float4 lg = *reinterpret_cast<const float4 *>(&sm.vlg[warp * 32 + r4]);
#pragma unroll
        for (int j = 0; j < HL; j++) {
            const float x = warp_max(fmaxf(fmaxf(__fadd_ru(s[0][j], lg.x), __fadd_ru(s[1][j], lg.y)), fmaxf(__fadd_ru(s[2][j], lg.z), __fadd_ru(s[3][j], lg.w))));
            if (lane < 4 && own) sm.red[hd + 4 * j][warp] = x;
        }
        if (more && tid == 0 && step + 1 >= it.t_hi) sm.next_j = drawn;
        sync();                                            // also: every thread is done with the K slots and weights
        const uint32_t startV = cur.startV >> 3;
        {
            bool n_on = true; int nb = b, nh = h, n_col = col, n_step = step + 1;      // the worker's next step (it may open the next column)
            if (n_step >= it.t_hi) {
                if (more) { have_next = item_of(P + sm.next_j, nit); if (!have_next) release(); }
                n_on = have_next && nit.t_lo < nit.t_hi;
                if (n_on) { n_col = nit.col; n_step = nit.t_lo; nb = n_col / Hkv; nh = n_col % Hkv; }
                if (have_next) q_fetch(nit.col);
            }
            // (its V units, on their way during the V phase, are first touched when it begins; this step's lie in shared memory)
            load_meta(n_on, nb, nh, n_col, n_step, cur);
            if (BULK && warp == 0) {                       // its K blocks land during the V phase
                if (__all_sync(0xffffffffu, k_landed)) stage_K(n_on, n_col, n_step);
                else if (lane == 0) sm.dead = 1;
            }
        }
        float alpha[HL], beta[HL];
        {
            const float4 sc = *reinterpret_cast<const float4 *>(&sm.vsc[warp * 32 + r4]), vz = *reinterpret_cast<const float4 *>(&sm.vz[warp * 32 + r4]);
            float u[HL];
            bool far = false;
#pragma unroll
            for (int j = 0; j < HL; j++) { u[j] = red_max(hd + 4 * j); far = far || fabsf(u[j]) >= FAR; }
            // the step's sums relative to e^u, and its V weights: the lane's four tokens are one word of its head
            auto put_weights = [&](int j, const float (&w)[4], float inv) {
                const uint2 w2 = pack_fix(w[0], w[1], w[2], w[3], inv);
                uint32_t *at = sm.w + 2 * VW + 2 * (hd + 4 * j) * COL_WORDS + warp * 8 + (lane >> 2);
                if (own) { at[0] = w2.x; at[COL_WORDS] = w2.y; }
            };
            auto weigh = [&](int j, float (&w)[4]) {
                const float m_new = fmaxf(m_run[j], u[j]);
                alpha[j] = exp_fast(m_run[j] - m_new); beta[j] = exp_fast(u[j] - m_new);    // exp(-inf) = 0 on the first step
                m_run[j] = m_new;
                const float p0 = exp_fast(s[0][j] - u[j]), p1 = exp_fast(s[1][j] - u[j]), p2 = exp_fast(s[2][j] - u[j]), p3 = exp_fast(s[3][j] - u[j]);
                l_run[j] = fmaf(l_run[j], alpha[j], beta[j] * ((p0 + p1) + (p2 + p3)));
                z_run[j] = fmaf(z_run[j], alpha[j], beta[j] * fmaf(p0, vz.x, fmaf(p1, vz.y, fmaf(p2, vz.z, p3 * vz.w))));
                w[0] = p0 * sc.x; w[1] = p1 * sc.y; w[2] = p2 * sc.z; w[3] = p3 * sc.w;
            };
            // (a warp holds all heads' maxima, so the worker's warps agree)
            if (!__any_sync(0xffffffffu, far)) {
#pragma unroll
                for (int j = 0; j < HL; j++) {
                    float w[4];
                    weigh(j, w);
                    beta[j] *= -1.0f / FIX_V;
                    put_weights(j, w, -FIX_V);
                }
            } else {
                float w[HL][4];
                sync();                                    // the maxima are read
#pragma unroll
                for (int j = 0; j < HL; j++) {
                    const float x = warp_max(fmaxf(fmaxf(s[0][j], s[1][j]), fmaxf(s[2][j], s[3][j])));
                    if (lane < 4 && own) sm.red[hd + 4 * j][warp] = x;
                }
                sync();
#pragma unroll
                for (int j = 0; j < HL; j++) { u[j] = red_max(hd + 4 * j); weigh(j, w[j]); }
                sync();
#pragma unroll
                for (int j = 0; j < HL; j++) {             // (a negative weight takes the shorter end of the range)
                    float x = 0.f;
#pragma unroll
                    for (int i = 0; i < 4; i++) x = fmaxf(x, fmaxf(w[j][i], -w[j][i] * (FIX_V / FIX_UP)));
                    x = warp_max(x);
                    if (lane < 4 && own) sm.red[hd + 4 * j][warp] = x;
                }
                sync();
#pragma unroll
                for (int j = 0; j < HL; j++) {
                    const float top = red_max(hd + 4 * j), inv = top > 0.f ? -FIX_V / top : 0.f;
#pragma unroll
                    for (int i = 0; i < 4; i++) w[j][i] = (float)__float2int_rn(w[j][i] * inv);       // (an infinite scale: no weight, and NaN through beta)
                    beta[j] *= top * (-1.0f / FIX_V);
                    put_weights(j, w[j], 1.0f);
                }
            }
        }
        v_landed = !BULK || kvc_mbar_wait(&sm.bar[1], par >> 1 & 1u, p.wait_limit);
        if (BULK && v_landed) par ^= 2u;
        if (!v_landed) flags |= KVC_FLAG_WAIT_TIMEOUT;
        v_staged = false;
        sync();
        // ---- V: this step's contribution to the lane's four channels
        {
            int d[4][HL];
            bool ok = v_landed && sm.okV[sub] && startV < sm.nbV[sub];
            // (and so does a warp whose lanes lag in two parts of four, for the rest of the item)
            uint32_t lagged = 0;
            const bool lone = (par & 4u) != 0;
            ok = rows_dot<G>(lone ? KvcWay{KVC_SINGLES, wayV.esc} : wayV, {kvc_smem_addr(slotsV + sub * p.slotV_bytes), ok ? sm.leadV[sub] + startV : 1u, lutV_s, loneV_s, tree_s + 2048u}, rows_s, kvc_smem_addr(sm.w + 2 * VW), lane, d, lagged) && ok;
            if (spare_in && lagged >= 2u) par |= 4u;
            if (!ok) flags |= KVC_FLAG_BAD_STREAM;
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < HL; j++) acc[i][j] = fmaf(acc[i][j], alpha[j], beta[j] * (float)d[i][j]);
        }
    }

    // ---- uncompressed tail, only for callers without a workspace: otherwise the merge kernel adds it
    if (p.Tr > 0 && !p.partial && (TEAM || it.t_hi == p.n_tiles)) {
        float *pt = reinterpret_cast<float *>(sm.w);       // p[row][g] of 128 rows
        for (long long r0 = TEAM ? wk % p.team * 128 : 0; r0 < p.Tr; r0 += TEAM ? p.team * 128 : 128) {      // a team's workers take the passes in turn
            const bool act = r0 + tid < p.Tr;
            sync();
            float s[G];
#pragma unroll
            for (int g = 0; g < G; g++) s[g] = act ? 0.f : -CUDART_INF_F;
            if (act) {
                const __half *kr = p.ktail + (((r0 + tid) * B + b) * Hkv + h) * 128;
#pragma unroll 1
                for (int c8 = 0; c8 < 16; c8++) {
                    uint4 kv = *reinterpret_cast<const uint4 *>(kr + c8 * 8);
                    const __half *kh = reinterpret_cast<const __half *>(&kv);
#pragma unroll
                    for (int k = 0; k < 8; k++)
#pragma unroll
                        for (int g = 0; g < G; g++) s[g] = fmaf(__half2float(kh[k]), sm.q[g * 128 + c8 * 8 + k], s[g]);
                }
            }
#pragma unroll
            for (int g = 0; g < G; g++) { const float mx = kvc_warp_max(s[g]); if (lane == 0) sm.red[g][warp] = mx; }
            sync();
            float alpha[HL], dv[4][HL];
#pragma unroll
            for (int j = 0; j < HL; j++) {
                const float m_new = fmaxf(m_run[j], red_max(hd + 4 * j));
                alpha[j] = exp_fast(m_run[j] - m_new);
                m_run[j] = m_new;
                if (tid < 4) sm.zp[hd + 4 * j] = m_new;
#pragma unroll
                for (int i = 0; i < 4; i++) dv[i][j] = 0.f;
            }
            sync();
#pragma unroll
            for (int g = 0; g < G; g++) {
                const float pr = act ? exp_fast(s[g] - sm.zp[g]) : 0.f;
                pt[tid * G + g] = pr;
                const float ssum = kvc_warp_sum(pr);
                if (lane == 0) sm.red[g][warp] = ssum;
            }
            sync();
            const int n_here = (int)min(128ll, p.Tr - r0);
            for (int i = 0; i < n_here; i++) {             // the lane's four channels over the pass's rows
                const __half *vr = p.vtail + (((r0 + i) * B + b) * Hkv + h) * 128 + warp * 32 + r4;
#pragma unroll
                for (int c = 0; c < 4; c++)
#pragma unroll
                    for (int j = 0; j < HL; j++) dv[c][j] = fmaf(pt[i * G + hd + 4 * j], __half2float(vr[c]), dv[c][j]);
            }
#pragma unroll
            for (int j = 0; j < HL; j++) {
                z_run[j] *= alpha[j];
                l_run[j] = fmaf(l_run[j], alpha[j], warp == 0 && r4 == 0 ? red_sum(hd + 4 * j) : 0.f);      // one of the lanes that are added up
#pragma unroll
                for (int c = 0; c < 4; c++) acc[c][j] = fmaf(acc[c][j], alpha[j], dv[c][j]);
            }
        }
    }
    if (it.t_lo >= it.t_hi && have_next) q_fetch(nit.col);     // an item without steps fetched nothing yet
    // the sums over the worker's tokens
    sync();                                                // (the tail's scratch and the last maxima are read)
#pragma unroll
    for (int j = 0; j < HL; j++) {
        const float l = warp_sum(l_run[j]), z = warp_sum(z_run[j]);
        if (lane < 4 && own) { sm.red[hd + 4 * j][warp] = l; sm.w[(hd + 4 * j) * 4 + warp] = __float_as_uint(z); }
    }
    sync();
#pragma unroll
    for (int j = 0; j < HL; j++) {
        l_run[j] = red_sum(hd + 4 * j);
        const float4 z = *reinterpret_cast<const float4 *>(&sm.w[(hd + 4 * j) * 4]);
#pragma unroll
        for (int i = 0; i < 4; i++) acc[i][j] += (z.x + z.y) + (z.z + z.w);
    }
    const long long head0 = (long long)b * Hq + (long long)h * Gt + p.g0;
    bool dead;
    if constexpr (TEAM) {                                  // each worker's share to its own shared memory, then a head per worker
        const int team = p.team, tm = wk / team, tk = wk % team;      // the worker's team and its place there
        auto team_sync = [&]() { asm volatile("bar.sync %0, %1;" :: "r"(rows_workers<G>() + 1 + tm), "r"(team * 128) : "memory"); };
        sync();                                            // (the sums are read)
        float *mine = reinterpret_cast<float *>(sm.w);     // acc[G][128]
#pragma unroll
        for (int j = 0; j < HL; j++) {
            if (!own) continue;
            *reinterpret_cast<float4 *>(mine + (hd + 4 * j) * 128 + warp * 32 + r4) = make_float4(acc[0][j], acc[1][j], acc[2][j], acc[3][j]);
            if (warp == 0 && lane < 4) { sm.red[hd + 4 * j][0] = m_run[j]; sm.red[hd + 4 * j][1] = l_run[j]; }
        }
        team_sync();
        const RowsWorker<G> *mates = &sm - tk;
        for (int g = tk; g < p.nh; g += team) {
            float M = -CUDART_INF_F, O = 0.f, L = 0.f;
            for (int w = 0; w < team; w++) M = fmaxf(M, mates[w].red[g][0]);
            for (int w = 0; w < team; w++) {
                const float m = mates[w].red[g][0], e = m == -CUDART_INF_F ? 0.f : exp_fast(m - M);     // a worker without tokens adds nothing
                L = fmaf(mates[w].red[g][1], e, L);
                O = fmaf(reinterpret_cast<const float *>(mates[w].w)[g * 128 + tid], e, O);
            }
            p.out[(head0 + g) * 128 + tid] = __float2half_rn(O / L);
        }
        dead = false;
        if (BULK) for (int w = 0; w < team; w++) dead |= mates[w].dead != 0;      // of any: a team stops together
        team_sync();
    } else {
#pragma unroll
    for (int j = 0; j < HL; j++) {
        if (!own || hd + 4 * j >= p.nh) continue;
        if (!p.partial) {
#pragma unroll
            for (int i = 0; i < 4; i++) p.out[(head0 + hd + 4 * j) * 128 + warp * 32 + r4 + i] = __float2half_rn(acc[i][j] / l_run[j]);
        } else {
            float *dst = p.ws_part + ((head0 + hd + 4 * j) * p.splits + it.part) * ROWS_PART_FLOATS;     // 8-byte aligned
            *reinterpret_cast<float2 *>(dst + 2 + warp * 32 + r4) = make_float2(acc[0][j], acc[1][j]);
            *reinterpret_cast<float2 *>(dst + 4 + warp * 32 + r4) = make_float2(acc[2][j], acc[3][j]);
            if (warp == 0 && lane < 4) { dst[0] = m_run[j]; dst[1] = l_run[j]; }
        }
    }
    sync();                                                // the sums are read before the next column's weights overwrite them
    dead = BULK && sm.dead != 0;
    }
    if (dead) break;                                       // a staging wait ran out: the status word says so, the item's result is void
    it = nit; have = have_next; have_next = false;
    if (!draw) have_next = have && item_of(++j_n1, nit);
    }   // items of the worker
    if (BULK && any) {                    // the copy of K issued after the last step is empty, but its phase must end;
        // after a wait that ran out, these are the phases still open: nothing may be in flight at the return
        if (!kvc_mbar_wait(&sm.bar[0], par & 1u, p.wait_limit)) flags |= KVC_FLAG_WAIT_TIMEOUT;
        if ((v_staged || !v_landed) && !kvc_mbar_wait(&sm.bar[1], par >> 1 & 1u, p.wait_limit)) flags |= KVC_FLAG_WAIT_TIMEOUT;
    }
    release();
    if (flags) atomicOr(p.status, flags);
    if (draw && tid == 0) {               // the last worker to finish leaves the scheduling counters zeroed for the next launch
        __threadfence();
        if (atomicAdd(&p.sched[1], 1) == P - 1) { p.sched[0] = 0; p.sched[1] = 0; __threadfence(); }
    }
}

// ---- one query head per KV head ------------------------------------------------------------------------
// The same workers with a decoder that multiplies as it goes: each lookup's symbols meet the weight record of its position
// (decode_dot), so there are no rows, and an SM holds one copy of the tables and up to ONE_WORKERS workers: 28 warps of 72
// registers where three CTAs of 256 threads with tables of their own, all eight warps at every barrier, were 24.  8 x 32 columns of
// 4096 tokens, rel 0.05 / 0.1: 135 us, now 128.  (Eight workers of 64 registers, 52 bytes of spills: 145, with runs of other lengths 134.)
constexpr int ONE_WORKERS = 7;

struct alignas(32) OneWorker {
    uint32_t w[2 * 2 * WROW];                // K weight records of the step's two blocks; scratch of the tail
    uint32_t ps_before[8];                   // bytes of the V records' neighbours ahead of the first one
    uint32_t ps[2 * WROW];                   // V weight records
    float red[4][4];                         // per-warp max, sum, zero-point and weight-max partials
    unsigned short q[128];                   // the query, fp16 bits
    float kstep[2], zp[2], qsum;
    uint64_t bar[2];                         // K and V staging barriers
    uint32_t leadK[4], leadV[4], nbK[4], nbV[4];   // of the two staged blocks (stage_bulk writes four entries)
    int okK[4], okV[4];
    int next_j, dead;
};
// tables, workers, slots (two of K and two of V each), bytes that a corrupt stream's overrun may read
size_t one_smem(const AttnParams &p, int workers) {
    return sizeof(OneTables) + workers * (sizeof(OneWorker) + 2 * (size_t)(p.slotK_bytes + p.slotV_bytes)) + SLOT_PAD;
}
int one_fit(const AttnParams &p) {
    int workers = ONE_WORKERS;
    while (workers > 1 && one_smem(p, workers) > MAX_CTA_SHARED) workers--;
    return workers;
}

// K weight records of block `sub`: lane = 4 consecutive channels; qh: the query's fp16 bits
__device__ __forceinline__ void k_weights_one(uint32_t *w, float *step, float *zp, const uint16_t *qh, float scaling, const KUnit &u,
                                              bool channel_units, int min_bytes, int sub, int lane) {
    const uint2 qb = *reinterpret_cast<const uint2 *>(qh + lane * 4);
    const uint32_t q2[2] = {qb.x, qb.y};
    float wv[4], z = 0.f;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float q = kvc_scale_value((unsigned short)(q2[i >> 1] >> (16 * (i & 1)))) * scaling, sc = kvc_scale_value(ku_scale(u, i));
        wv[i] = q * sc;
        z = fmaf((float)ku_min(u, i, min_bytes) * sc, q, z);
    }
    const float mx = kvc_warp_max(fmaxf(fmaxf(fabsf(wv[0]), fabsf(wv[1])), fmaxf(fabsf(wv[2]), fabsf(wv[3]))));
    z = channel_units ? kvc_warp_sum(z) : 0.f;
    const float st = fix_step(mx), inv = st > 0.f ? 1.0f / st : 0.f;
    int q4[7];
#pragma unroll
    for (int i = 0; i < 4; i++) q4[i] = __float2int_rn(wv[i] * inv);
#pragma unroll
    for (int i = 0; i < 3; i++) {                               // the next lane's first three values
        const int nv = __shfl_down_sync(0xffffffffu, q4[i], 1);
        q4[4 + i] = lane == 31 ? 0 : nv;
    }
    uint32_t *row = w + sub * 2 * WROW;
#pragma unroll
    for (int i = 0; i < 4; i += 2) {
        const uint2 a = pack4(q4[i], q4[i + 1], q4[i + 2], 0), b = pack4(q4[i + 1], q4[i + 2], q4[i + 3], 0);
        *reinterpret_cast<uint4 *>(&row[2 * (lane * 4 + i)]) = make_uint4(a.x, a.y, b.x, b.y);
    }
    if (lane < 2 * (WROW - 128)) row[2 * 128 + lane] = 0u;
    if (lane == 0) { step[sub] = st; zp[sub] = z; }
}

__device__ __forceinline__ void sts8(uint32_t addr, uint32_t v) { asm volatile("st.shared.u8 [%0], %1;" :: "r"(addr), "r"(v) : "memory"); }

template <bool BULK, bool TEAM>
__global__ void __launch_bounds__(128 * ONE_WORKERS, 1) attn_one_kernel(AttnParams p) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    OneTables &tab = *reinterpret_cast<OneTables *>(smem_raw);
    const int workers = blockDim.x >> 7, wk = threadIdx.x >> 7;
    const int tid = threadIdx.x & 127, lane = tid & 31, warp = tid >> 5, sub = tid >> 6, v = tid & 63;
    uint8_t *const wbase = smem_raw + sizeof(OneTables), *const sbase = wbase + workers * sizeof(OneWorker);
    OneWorker &sm = reinterpret_cast<OneWorker *>(wbase)[wk];
    uint8_t *const slotsK = sbase + wk * 2 * (p.slotK_bytes + p.slotV_bytes), *const slotsV = slotsK + 2 * p.slotK_bytes;
    auto sync = [&]() { asm volatile("bar.sync %0, 128;" :: "r"(wk + 1) : "memory"); };     // the worker's threads
    auto release = []() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); };
    // launched with programmatic stream serialisation, as the grouped kernel: set-up before griddepcontrol.wait reads cache data only
    const int B = (int)p.B, Hkv = (int)p.Hkv, cols = B * Hkv;
    const kvc_qmeta_dev &km = p.k.q, &vm = p.v.q;
    int flags = 0;

    struct Item { int col, t_lo, t_hi, part; };            // steps t_lo .. t_hi - 1 of a column; part: the run's index
    const bool draw = !TEAM && p.sched != nullptr;
    const int P = (int)gridDim.x * (TEAM ? workers / p.team : workers);
    const int me = TEAM ? wk / p.team * (int)gridDim.x + (int)blockIdx.x : (int)blockIdx.x * workers + wk;
    const int w_hi = draw ? (int)p.work : (int)(p.work * (me + 1) / P);
    auto item_of = [&](int j, Item &it) -> bool {
        if (j >= w_hi) return false;
        const int n_long = cols * p.long_runs;
        if constexpr (TEAM) {                              // the worker's share of column j: the same for every column
            const int tk = wk % p.team;
            it.col = j; it.part = 0; it.t_lo = (int)((long long)p.n_tiles * tk / p.team); it.t_hi = (int)((long long)p.n_tiles * (tk + 1) / p.team);
        } else if (j < n_long) {
            const int r = j % p.long_runs;
            it.col = j / p.long_runs; it.part = r; it.t_lo = r * p.tiles_per_split; it.t_hi = min(p.n_tiles, it.t_lo + p.tiles_per_split);
        } else {
            const int n_short = p.splits - p.long_runs, r = (j - n_long) % n_short;
            it.col = (j - n_long) / n_short; it.part = p.long_runs + r;
            it.t_lo = p.long_runs * p.tiles_per_split + r * p.short_tiles; it.t_hi = min(p.n_tiles, it.t_lo + p.short_tiles);
        }
        return true;
    };
    auto blkK_of = [&](int col, int t, int l) { return ((long long)t * 2 + l) * cols + col; };
    auto blkV_of = [&](int col, int t, int l) { return (long long)t * (cols * 2) + (long long)col * 2 + l; };

    Item it, nit;
    int j_n1 = draw ? P + me : (int)(p.work * me / P) + 1;
    bool have = item_of(draw ? me : j_n1 - 1, it), have_next = have && item_of(j_n1, nit);
    int drawn = 0;                                         // thread 0: the counter's answer, used an item later
    const bool any = have && it.t_lo < it.t_hi;

    // the two blocks of a step, by the lanes 0 and 1 of the worker's first warp
    auto stage_K = [&](bool on, int col, int t) { stage_bulk(p.k, on && lane < 2, blkK_of(col, t, lane & 1), slotsK + (lane & 1) * p.slotK_bytes, sm.leadK, sm.okK, sm.nbK, &sm.bar[0], lane, p.starve != 0); };
    auto stage_V = [&](bool on, int col, int t) { stage_bulk(p.v, on && lane < 2, blkV_of(col, t, lane & 1), slotsV + (lane & 1) * p.slotV_bytes, sm.leadV, sm.okV, sm.nbV, &sm.bar[1], lane, p.starve != 0); };
    if (BULK) {
        if (tid == 0) { kvc_mbar_init(&sm.bar[0], 1); kvc_mbar_init(&sm.bar[1], 1); kvc_mbar_fence_init(); sm.dead = 0; }
        sync();
        if (warp == 0 && any) { stage_K(true, it.col, it.t_lo); stage_V(true, it.col, it.t_lo); }
    }
    kvc_load_luts(tab.lutK, tab.lutV, p.k.book, p.v.book, threadIdx.x, blockDim.x);
    const bool escK = book_has_long_codes(p.k.book), escV = book_has_long_codes(p.v.book);
    for (int i = tid; i < 2 * WROW; i += 128) sm.ps[i] = 0u;   // V records: the bytes that no token writes stay zero

    struct StepMeta { unsigned short startK, startV, vsc, ksc; int vmi, kmi; KUnit ku; };   // as loaded: no arithmetic waits on them here
    auto load_meta = [&](bool on, int col, int step, StepMeta &m) {
        const long long t = (long long)step * 128 + tid;
        const int b = col / Hkv, h = col % Hkv;
        m.startK = m.startV = 0; m.vsc = 0; m.vmi = m.kmi = 0; m.ksc = 0x3c00;
        m.ku.sc = make_uint2(0x3c003c00u, 0x3c003c00u); m.ku.mi = make_uint2(0u, 0u);          // 1.0, 0
        if (!on) return;
        m.startK = vec_start_bits(p.k.thread_info, blkK_of(col, step, sub), v);
        m.startV = vec_start_bits(p.v.thread_info, blkV_of(col, step, sub), v);
        const long long u = kvc_tok_unit(t, vm.tok_div) * vm.sj + b * vm.sb + h * vm.sh;
        m.vsc = kvc_load_scale_bits(vm, u); m.vmi = kvc_load_min(vm, u);
        if (km.sc == 0) k_token_unit(m.ksc, m.kmi, km, t, b, h);
        else if (warp < 2) {                               // of the block whose weights the warp builds, 4 channels per lane
            const long long un = kvc_tok_unit((long long)step * 128 + warp * 64, km.tok_div) * km.sj + b * km.sb + h * km.sh + lane * 4;
            m.ku.sc = *reinterpret_cast<const uint2 *>(reinterpret_cast<const unsigned short *>(km.scale) + un);
            if (km.min_bytes == 1) m.ku.mi.x = *reinterpret_cast<const uint32_t *>(reinterpret_cast<const int8_t *>(km.min_int) + un);
            else m.ku.mi = *reinterpret_cast<const uint2 *>(reinterpret_cast<const int16_t *>(km.min_int) + un);
        }
    };
    StepMeta cur, nxt;
    load_meta(any, have ? it.col : 0, have ? it.t_lo : 0, cur);
    unsigned short qn = 0;                                 // the query of an item is fetched while the item before it runs; a column is a head
    auto q_fetch = [&](int col_) { qn = reinterpret_cast<const unsigned short *>(p.q)[(long long)col_ * 128 + tid]; };
    __syncthreads();                                       // the tables are in; from here on the workers go their own ways
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (have) q_fetch(it.col);

    uint32_t par = 0;                                      // bit 0 / bit 1: parity of the staging phase the K / V barrier is waited for next
    while (have) {
    const int col = it.col, b = col / Hkv, h = col % Hkv;
    if (!have_next && p.early) release();
    if (draw && tid == 0) drawn = atomicAdd(&p.sched[0], 1);
    sm.q[tid] = qn;
    sync();
    if (warp == 3) {                                       // sum of the query's 128 (scaled) values (read behind the next barrier)
        float a = 0.f;
#pragma unroll
        for (int k = 0; k < 4; k++) a += kvc_scale_value(sm.q[k * 32 + lane]) * p.scaling;
        a = kvc_warp_sum(a);
        if (lane == 0) sm.qsum = a;
    }
    float m_run = -CUDART_INF_F, l_run = 0.f, acc = 0.f;   // acc: channel tid

    for (int step = it.t_lo; step < it.t_hi; step++) {
        bool n_on = true; int n_col = col, n_step = step + 1;      // the worker's next step (it may open the next column)
        if (n_step >= it.t_hi) {
            n_on = have_next && nit.t_lo < nit.t_hi; n_col = n_on ? nit.col : col; n_step = n_on ? nit.t_lo : 0;
            if (have_next) q_fetch(nit.col);
        }
        if (!BULK) {
            uint32_t ld, nb;
            bool ok = stage(p.k, blkK_of(col, step, sub), slotsK + sub * p.slotK_bytes, &ld, &nb, v);
            if (v == 0) { sm.leadK[sub] = ld; sm.nbK[sub] = nb; sm.okK[sub] = ok; }
            ok = stage(p.v, blkV_of(col, step, sub), slotsV + sub * p.slotV_bytes, &ld, &nb, v);
            if (v == 0) { sm.leadV[sub] = ld; sm.nbV[sub] = nb; sm.okV[sub] = ok; }
        }
        if (warp < 2) k_weights_one(sm.w, sm.kstep, sm.zp, sm.q, p.scaling, cur.ku, km.sc != 0, km.min_bytes, warp, lane);
        // A wait that runs out: the thread does not decode.  The warp that issues the copies looks at its own verdict: a barrier
        // whose phase it did not see complete is never armed again (a second arrival on an open phase is an error), and the worker
        // is marked; it takes no further item, and what it had in flight is waited for once more, bounded, before it returns.
        bool k_landed = true;
        if (BULK) {
            k_landed = kvc_mbar_wait(&sm.bar[0], par & 1u, p.wait_limit);
            if (k_landed) par ^= 1u; else flags |= KVC_FLAG_WAIT_TIMEOUT;
        }
        sync();
        // ---- K: the score of the thread's token
        float s;
        {
            int hi[1] = {0}, lo[1] = {0};
            bool ok = k_landed && sm.okK[sub] && (uint32_t)(cur.startK >> 3) < sm.nbK[sub];      // a vector begins inside its block
            if (ok) {
                const uint32_t slot_s = kvc_smem_addr(slotsK + sub * p.slotK_bytes), at = sm.leadK[sub] + (cur.startK >> 3), w_s = kvc_smem_addr(sm.w + sub * 2 * WROW);
                ok = escK ? decode_dot_impl<1, true>(slot_s, at, kvc_smem_addr(tab.lutK), KvcTreeGlobal(p.k.book), w_s, hi, lo)
                          : decode_dot_impl<1, false>(slot_s, at, kvc_smem_addr(tab.lutK), KvcTreeGlobal(p.k.book), w_s, hi, lo);
            }
            if (!ok) flags |= KVC_FLAG_BAD_STREAM;
            const float d = fix_value(sm.kstep[sub], hi[0], lo[0]);
            s = km.sc != 0 ? d + sm.zp[sub] : kvc_scale_value(cur.ksc) * fmaf((float)cur.kmi, sm.qsum, d);
        }
        // ---- online softmax over the step
        {
            const float mx = kvc_warp_max(s);
            if (lane == 0) sm.red[0][warp] = mx;
        }
        sync();                                            // also: every thread is done with the K slots and weights
        load_meta(n_on, n_col, n_step, nxt);               // in flight during the V phase, first touched in the next step
        if (BULK && warp == 0) {                           // the next step's K blocks land during the V phase
            if (__all_sync(0xffffffffu, k_landed)) stage_K(n_on, n_col, n_step);
            else if (lane == 0) sm.dead = 1;
        }
        float alpha, wv;
        {
            const float4 x = *reinterpret_cast<const float4 *>(sm.red[0]);
            const float m_new = fmaxf(fmaxf(m_run, fmaxf(x.x, x.y)), fmaxf(x.z, x.w));
            alpha = __expf(m_run - m_new);                 // exp(-inf) = 0 on the first step
            m_run = m_new;
            const float pr = __expf(s - m_new);
            wv = pr * kvc_scale_value(cur.vsc);
            const float ssum = kvc_warp_sum(pr), zsum = kvc_warp_sum(wv * (float)cur.vmi), wmax = kvc_warp_max(fabsf(wv));
            if (lane == 0) { sm.red[1][warp] = ssum; sm.red[2][warp] = zsum; sm.red[3][warp] = wmax; }
        }
        sync();
        // The V weights: the token's 16-bit value is a byte of either word of three records -- its own, and those of the two
        // positions ahead of it (no exchange of values, no barrier for one).
        float vst;
        {
            const float4 x = *reinterpret_cast<const float4 *>(sm.red[3]);
            vst = fix_step(fmaxf(fmaxf(x.x, x.y), fmaxf(x.z, x.w)));
            const int q16 = __float2int_rn(wv * (vst > 0.f ? 1.0f / vst : 0.f));
            const uint32_t a = kvc_smem_addr(sm.ps) + tid * 8, qh = (uint32_t)q16 >> 8, ql = (uint32_t)q16;
            sts8(a + 1, qh); sts8(a + 5, ql); sts8(a - 6, qh); sts8(a - 2, ql); sts8(a - 13, qh); sts8(a - 9, ql);
        }
        const bool v_landed = !BULK || kvc_mbar_wait(&sm.bar[1], par >> 1, p.wait_limit);
        if (BULK && v_landed) par ^= 2u;
        if (!v_landed) flags |= KVC_FLAG_WAIT_TIMEOUT;
        sync();
        // ---- V: this step's contribution to the thread's channel
        {
            int hi[1] = {0}, lo[1] = {0};
            bool ok = v_landed && sm.okV[sub] && (uint32_t)(cur.startV >> 3) < sm.nbV[sub];
            if (ok) {
                const uint32_t slot_s = kvc_smem_addr(slotsV + sub * p.slotV_bytes), at = sm.leadV[sub] + (cur.startV >> 3), w_s = kvc_smem_addr(sm.ps);
                ok = escV ? decode_dot_impl<1, true>(slot_s, at, kvc_smem_addr(tab.lutV), KvcTreeGlobal(p.v.book), w_s, hi, lo)
                          : decode_dot_impl<1, false>(slot_s, at, kvc_smem_addr(tab.lutV), KvcTreeGlobal(p.v.book), w_s, hi, lo);
            }
            if (!ok) flags |= KVC_FLAG_BAD_STREAM;
            const float4 x = *reinterpret_cast<const float4 *>(sm.red[1]), z = *reinterpret_cast<const float4 *>(sm.red[2]);
            l_run = l_run * alpha + ((x.x + x.y) + (x.z + x.w));
            acc = fmaf(acc, alpha, fix_value(vst, hi[0], lo[0]) + ((z.x + z.y) + (z.z + z.w)));
        }
        sync();                                            // every thread is done with the V slots, weights and sums
        if (BULK && warp == 0) {                           // the next step's V blocks land during its K phase
            if (__all_sync(0xffffffffu, v_landed)) stage_V(n_on, n_col, n_step);
            else if (lane == 0) sm.dead = 1;
        }
        cur = nxt;
    }

    // ---- uncompressed tail, only for callers without a workspace: otherwise the merge kernel adds it
    if (p.Tr > 0 && !p.partial && (TEAM || it.t_hi == p.n_tiles)) {
        float *pt = reinterpret_cast<float *>(sm.w);       // p of 128 rows
        for (long long r0 = TEAM ? wk % p.team * 128 : 0; r0 < p.Tr; r0 += TEAM ? p.team * 128 : 128) {      // a team's workers take the passes in turn
            const bool act = r0 + tid < p.Tr;
            sync();
            float s = -CUDART_INF_F;
            if (act) {
                s = 0.f;
                const __half *kr = p.ktail + (((r0 + tid) * B + b) * Hkv + h) * 128;
#pragma unroll 1
                for (int c8 = 0; c8 < 16; c8++) {
                    const uint4 kv = *reinterpret_cast<const uint4 *>(kr + c8 * 8);
                    const __half *kh = reinterpret_cast<const __half *>(&kv);
#pragma unroll
                    for (int k = 0; k < 8; k++) s = fmaf(__half2float(kh[k]), kvc_scale_value(sm.q[c8 * 8 + k]) * p.scaling, s);
                }
            }
            const float mx = kvc_warp_max(s);
            if (lane == 0) sm.red[0][warp] = mx;
            sync();
            const float4 x = *reinterpret_cast<const float4 *>(sm.red[0]);
            const float m_new = fmaxf(fmaxf(m_run, fmaxf(x.x, x.y)), fmaxf(x.z, x.w)), alpha = __expf(m_run - m_new);
            m_run = m_new;
            const float pr = act ? __expf(s - m_new) : 0.f;
            pt[tid] = pr;
            const float ssum = kvc_warp_sum(pr);
            if (lane == 0) sm.red[1][warp] = ssum;
            sync();
            const int n_here = (int)min(128ll, p.Tr - r0);
            float dv = 0.f;
            for (int i = 0; i < n_here; i++) dv = fmaf(pt[i], __half2float(p.vtail[(((r0 + i) * B + b) * Hkv + h) * 128 + tid]), dv);
            const float4 y = *reinterpret_cast<const float4 *>(sm.red[1]);
            l_run = l_run * alpha + ((y.x + y.y) + (y.z + y.w));
            acc = fmaf(acc, alpha, dv);
        }
    }
    if (it.t_lo >= it.t_hi && have_next) q_fetch(nit.col);     // an item without steps fetched nothing yet
    bool dead;
    if constexpr (TEAM) {                                  // each worker's share to its own shared memory, then the sum
        const int team = p.team, tm = wk / team, tk = wk % team;      // the worker's team and its place there
        auto team_sync = [&]() { asm volatile("bar.sync %0, %1;" :: "r"(ONE_WORKERS + 1 + tm), "r"(team * 128) : "memory"); };
        sync();                                            // (the tail's scratch is read)
        reinterpret_cast<float *>(sm.w)[tid] = acc;
        if (tid == 0) { sm.red[0][0] = m_run; sm.red[0][1] = l_run; }
        team_sync();
        const OneWorker *mates = &sm - tk;
        if (tk == 0) {
            float M = -CUDART_INF_F, O = 0.f, L = 0.f;
            for (int w = 0; w < team; w++) M = fmaxf(M, mates[w].red[0][0]);
            for (int w = 0; w < team; w++) {
                const float m = mates[w].red[0][0], e = m == -CUDART_INF_F ? 0.f : __expf(m - M);     // a worker without tokens adds nothing
                L = fmaf(mates[w].red[0][1], e, L);
                O = fmaf(reinterpret_cast<const float *>(mates[w].w)[tid], e, O);
            }
            p.out[(long long)col * 128 + tid] = __float2half_rn(O / L);
        }
        dead = false;
        if (BULK) for (int w = 0; w < team; w++) dead |= mates[w].dead != 0;      // of any: a team stops together
        team_sync();
    } else {
        if (!p.partial) p.out[(long long)col * 128 + tid] = __float2half_rn(acc / l_run);
        else {
            float *dst = p.ws_part + ((long long)col * p.splits + it.part) * ROWS_PART_FLOATS;
            dst[2 + tid] = acc;
            if (tid == 0) { dst[0] = m_run; dst[1] = l_run; }
        }
        if (draw && tid == 0) sm.next_j = drawn;
        sync();                                            // the tail's scratch is read before the next column's weights overwrite it
        dead = BULK && sm.dead != 0;
    }
    if (dead) break;                                       // a staging wait ran out: the status word says so, the item's result is void
    const int j_n2 = draw ? 2 * P + sm.next_j : j_n1 + 1;
    it = nit; have = have_next; j_n1 = j_n2;
    have_next = have && item_of(j_n1, nit);
    }   // items of the worker
    if (BULK && any) {                    // the copies issued after the last step are empty, but their phase must end;
        // after a wait that ran out, these are the phases still open: nothing may be in flight at the return
        if (!kvc_mbar_wait(&sm.bar[0], par & 1u, p.wait_limit)) flags |= KVC_FLAG_WAIT_TIMEOUT;
        if (!kvc_mbar_wait(&sm.bar[1], par >> 1, p.wait_limit)) flags |= KVC_FLAG_WAIT_TIMEOUT;
    }
    release();
    if (flags) atomicOr(p.status, flags);
    if (draw && tid == 0) {               // the last worker to finish leaves the scheduling counters zeroed for the next launch
        __threadfence();
        if (atomicAdd(&p.sched[1], 1) == P - 1) { p.sched[0] = 0; p.sched[1] = 0; __threadfence(); }
    }
}

// The uncompressed tail of a cache (the recent window): dense fp16 rows [Tr, B, Hkv, 128] behind the compressed part.
struct TailArgs {
    const __half *q, *ktail, *vtail;
    long long Tr;
    int B, Hkv, Hq;
    float scaling;
};

// Loads that stay where they are written: a batch of them is issued before the first use (left to itself the
// compiler moves each load down to its use, and the batch becomes a chain of memory round trips).
__device__ __forceinline__ uint4 ld_nc_128_pinned(const void *p) {
    uint4 v;
    asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t ld_nc_32_pinned(const void *p) {
    uint32_t v;
    asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ unsigned short ld_nc_16_pinned(const void *p) {
    unsigned short v;
    asm volatile("ld.global.nc.u16 %0, [%1];" : "=h"(v) : "l"(p));
    return v;
}

// Merges the `splits` partial results of every head and adds the tail: grid = heads; 256 threads: the first 128 are the output channels.
//
// The tail is this kernel's work, not the attention kernel's: its rows lie a whole token row apart in memory, so
// every step of it (the query, the K rows, the V rows) is a round trip to memory with little to do in between.
// Inside the attention kernel each column's tail held a 256-thread CTA and its third of an SM for those round
// trips (a 128-row tail lengthened a 137 us launch by 160 us when its loads depended on one another, by 25 us
// with deep batches).  Here every head's tail is in flight at once on small CTAs, and it runs before the
// grid-dependency wait, i.e. while the attention kernel's last CTAs still work: it reads nothing that kernel writes, and
// that kernel has itself waited for whatever wrote the query and the tail's rows.  With nothing compressed (splits = 0)
// there is no attention kernel in between: the kernel ahead may be the one that stores the newest rows (it lets its
// dependents start early), so the wait comes first.
// The loads of the partial results are issued in batches of 16 before any is used as well, by both halves of the CTA in turn:
// (2 columns of 32768 tokens, 2 heads each, 256 partial results: 32.5 us for the step with batches of 8 by one half, now 24.5).
constexpr int MERGE_THREADS = 256;
// PAIRS: the tail's rows of V start on 4 bytes (else on 2: a load per channel).  REGS: with 96 registers a CTA finds room beside three workers of the grouped kernel or four
// with one head, with 128 it stays off their SM: which is better as long as the SMs without attention CTAs, two a piece, hold them all, as company slows the workers.  (10 columns of 5376 tokens and 152
// rows, 3 heads, 140 attention CTAs and 30 of this kernel: 23.3 and 17.1 us; 12 of 2816 and 165, 6 heads, 132 and 72: 16.9 and 16.3; 32 of 1792 and 208, one head, 112 and 32: 14.0 and 15.0.)
template <bool PAIRS, int REGS>
__global__ void __maxnreg__(REGS) attn_merge_kernel(const float *__restrict__ ws_part, __half *__restrict__ out, int splits, TailArgs t) {
    __shared__ float sm_red[8], sm_sum[8];
    __shared__ __align__(16) float sm_e[128], sm_o[512];
    __shared__ __align__(16) float sm_q[128];
    constexpr int PART = ROWS_PART_FLOATS;
    const float *src = ws_part + (size_t)blockIdx.x * splits * PART;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // launched with programmatic stream serialisation: the kernel behind this one in the stream may set up
    // while this one runs (it touches nothing this one writes before its own wait), and this one's CTAs may be
    // resident before the attention kernel has finished; its partial results are complete and visible after the wait
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (splits == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
    float m_t = -CUDART_INF_F, l_t = 0.f, o_t = 0.f;      // the tail's running maximum and sum; its output of channel tid (of the first 128 threads)
    if (t.Tr > 0) {
        // q.k: two threads per row, 64 channels each; P.V: thread = (quarter of the pass's rows, two channels).  (With a channel and half of
        // the rows it took 128 registers.)
        const int row = tid >> 1, part = tid & 1, ch = (tid & 63) * 2, rg = tid >> 6;
        const long long b = blockIdx.x / t.Hq, h = (blockIdx.x % t.Hq) / (t.Hq / t.Hkv);
        const long long rstride = (long long)t.B * t.Hkv * 128;                 // halves between two rows of a column
        const __half *kcol = t.ktail + (b * t.Hkv + h) * 128 + part * 64, *vcol = t.vtail + (b * t.Hkv + h) * 128 + ch;
        // Every load of a pass -- the query (first pass), the thread's half row of K, its 32 rows of V -- is issued
        // before the first of them is used: one trip to memory per pass instead of one per step of the softmax.
        float o0 = 0.f, o1 = 0.f;                                             // the thread's two channels over its rows
        const unsigned short qbits = tid < 128 ? ld_nc_16_pinned(t.q + (size_t)blockIdx.x * 128 + tid) : (unsigned short)0;
        for (long long r0 = 0; r0 < t.Tr; r0 += 128) {                        // 128 rows per pass
            const int n_here = (int)min(128ll, t.Tr - r0);
            const bool act = row < n_here;
            uint4 kv[8];
            const __half *kr = kcol + (r0 + min(row, n_here - 1)) * rstride;  // rows beyond the pass: read again, not used
#pragma unroll
            for (int j = 0; j < 8; j++) kv[j] = ld_nc_128_pinned(kr + j * 8);
            uint32_t vv[32];
            const __half *vr = vcol + r0 * rstride;
            if (PAIRS) {
#pragma unroll
                for (int k = 0; k < 32; k++) vv[k] = ld_nc_32_pinned(vr + min(rg * 32 + k, n_here - 1) * rstride);   // rows beyond the pass: weight 0
            } else {
#pragma unroll
                for (int k = 0; k < 32; k++) {
                    const __half *x = vr + min(rg * 32 + k, n_here - 1) * rstride;
                    vv[k] = (uint32_t)ld_nc_16_pinned(x) | (uint32_t)ld_nc_16_pinned(x + 1) << 16;
                }
            }
            if (r0 == 0 && tid < 128) sm_q[tid] = __half2float(__ushort_as_half(qbits)) * t.scaling;
            __syncthreads();                                                  // sm_q is written; the pass before is done with sm_e
            float sc = -CUDART_INF_F;
            if (act) {
                float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;                 // four sums: no chain of 64 dependent additions
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const __half2 *kh = reinterpret_cast<const __half2 *>(&kv[j]);
                    const float4 q0 = *reinterpret_cast<const float4 *>(&sm_q[part * 64 + j * 8]);
                    const float4 q1 = *reinterpret_cast<const float4 *>(&sm_q[part * 64 + j * 8 + 4]);
                    const float2 k0 = __half22float2(kh[0]), k1 = __half22float2(kh[1]), k2 = __half22float2(kh[2]), k3 = __half22float2(kh[3]);
                    a0 = fmaf(k0.x, q0.x, a0); a1 = fmaf(k0.y, q0.y, a1); a2 = fmaf(k1.x, q0.z, a2); a3 = fmaf(k1.y, q0.w, a3);
                    a0 = fmaf(k2.x, q1.x, a0); a1 = fmaf(k2.y, q1.y, a1); a2 = fmaf(k3.x, q1.z, a2); a3 = fmaf(k3.y, q1.w, a3);
                }
                sc = (a0 + a1) + (a2 + a3);
            }
            const float other = __shfl_xor_sync(0xffffffffu, sc, 1);          // the row's other half (both -inf beyond the tail)
            sc = act ? sc + other : sc;
            const float mx = kvc_warp_max(sc);
            if (lane == 0) sm_red[warp] = mx;
            __syncthreads();
            float mt = sm_red[0];
#pragma unroll
            for (int w = 1; w < 8; w++) mt = fmaxf(mt, sm_red[w]);
            const float m_new = fmaxf(m_t, mt);
            const float alpha = __expf(m_t - m_new);                          // exp(-inf) = 0 in the first pass
            const float pr = act ? __expf(sc - m_new) : 0.f;
            if (part == 0) sm_e[row] = pr;
            const float ps = kvc_warp_sum(part == 0 ? pr : 0.f);
            if (lane == 0) sm_sum[warp] = ps;
            __syncthreads();
            float lsum = 0.f;
#pragma unroll
            for (int w = 0; w < 8; w++) lsum += sm_sum[w];
            l_t = l_t * alpha + lsum;
            m_t = m_new;
            float d0 = 0.f, d1 = 0.f, d2 = 0.f, d3 = 0.f;                     // rows rg * 32 .. + 31 of the pass, two sums per channel
#pragma unroll
            for (int k = 0; k < 32; k += 2) {
                const float2 x = __half22float2(*reinterpret_cast<const __half2 *>(&vv[k])), y = __half22float2(*reinterpret_cast<const __half2 *>(&vv[k + 1]));
                const float2 e = *reinterpret_cast<const float2 *>(&sm_e[rg * 32 + k]);
                d0 = fmaf(e.x, x.x, d0); d1 = fmaf(e.x, x.y, d1);
                d2 = fmaf(e.y, y.x, d2); d3 = fmaf(e.y, y.y, d3);
            }
            o0 = fmaf(o0, alpha, d0 + d2); o1 = fmaf(o1, alpha, d1 + d3);
        }
        __syncthreads();                                                      // sm_red and sm_e serve the merge below
        *reinterpret_cast<float2 *>(&sm_o[rg * 128 + ch]) = make_float2(o0, o1);
        __syncthreads();
        if (tid < 128) o_t = (sm_o[tid] + sm_o[128 + tid]) + (sm_o[256 + tid] + sm_o[384 + tid]);
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    constexpr int BATCH = 16;                             // partial results whose channel a thread loads at once, the CTA's two halves in turn
    const int c = tid & 127;
    float O = 0.f, L = 0.f;                               // O: channel tid & 127
    float M = -CUDART_INF_F;                              // the maximum over all partial results
    if (splits <= 128) {
        // Everything the first 32 partial results hold, and all maxima and sums, in one trip to memory: 0.7 us less where each was a trip of its own.
        float m2 = -CUDART_INF_F, l2 = 0.f, a[BATCH];
        if (tid < splits) { m2 = src[(size_t)tid * PART]; l2 = src[(size_t)tid * PART + 1]; }
        const int i0 = (tid >> 7) * BATCH;
#pragma unroll
        for (int k = 0; k < BATCH; k++) if (i0 + k < splits) a[k] = src[(size_t)(i0 + k) * PART + 2 + c];
        M = kvc_warp_max(m2);
        if (lane == 0) sm_red[warp] = M;
        __syncthreads();
        M = m_t;
#pragma unroll
        for (int w = 0; w < 8; w++) M = fmaxf(M, sm_red[w]);
        if (tid < 128) {
            const float e = m2 == -CUDART_INF_F ? 0.f : __expf(m2 - M);
            L = l2 * e;
            sm_e[tid] = e;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BATCH; k++) if (i0 + k < splits) O = fmaf(a[k], sm_e[i0 + k], O);
        for (int i1 = i0 + 2 * BATCH; i1 < splits; i1 += 2 * BATCH) {
#pragma unroll
            for (int k = 0; k < BATCH; k++) a[k] = src[(size_t)min(i1 + k, splits - 1) * PART + 2 + c];
#pragma unroll
            for (int k = 0; k < BATCH; k++) if (i1 + k < splits) O = fmaf(a[k], sm_e[i1 + k], O);
        }
    } else {
    for (int s2 = tid; s2 < splits; s2 += MERGE_THREADS) M = fmaxf(M, src[(size_t)s2 * PART]);
    M = kvc_warp_max(M);
    if (lane == 0) sm_red[warp] = M;
    __syncthreads();
    M = m_t;
#pragma unroll
    for (int w = 0; w < 8; w++) M = fmaxf(M, sm_red[w]);
    for (int s0 = 0; s0 < splits; s0 += 128) {
        const int ns = min(128, splits - s0);
        __syncthreads();                                  // the weights of the batch before are spent
        if (tid < 128) {
            float e = 0.f;
            if (tid < ns) {
                const float *pp = src + (size_t)(s0 + tid) * PART;
                const float m2 = pp[0];
                e = m2 == -CUDART_INF_F ? 0.f : __expf(m2 - M);
                L = fmaf(pp[1], e, L);
            }
            sm_e[tid] = e;
        }
        __syncthreads();
        // channel c of BATCH partial results, all loads in flight together
        for (int i0 = (tid >> 7) * BATCH; i0 < ns; i0 += 2 * BATCH) {
            float a[BATCH];
#pragma unroll
            for (int k = 0; k < BATCH; k++) {
                const float *pp = src + (size_t)(s0 + min(i0 + k, ns - 1)) * PART;
                a[k] = pp[2 + c];
            }
#pragma unroll
            for (int k = 0; k < BATCH; k++) if (i0 + k < ns) O = fmaf(a[k], sm_e[i0 + k], O);
        }
    }
    }
    if (tid >= 128) sm_o[tid - 128] = O;                  // the second half's sum joins the first's
    L = kvc_warp_sum(L);
    __syncthreads();
    if (lane == 0) sm_red[warp] = L;
    __syncthreads();
    L = 0.f;
#pragma unroll
    for (int w = 0; w < 4; w++) L += sm_red[w];           // warps 0..3 hold the partial results' sums
    if (tid < 128) O += sm_o[tid];
    const float e_t = m_t == -CUDART_INF_F ? 0.f : __expf(m_t - M);
    O = fmaf(o_t, e_t, O);
    L = fmaf(l_t, e_t, L);
    if (tid < 128) out[(size_t)blockIdx.x * 128 + tid] = __float2half_rn(O / L);
}

// Launch with programmatic stream serialisation: the grid may be set up on the device while the kernel
// ahead of it in the stream still runs.  Such a kernel starts with griddepcontrol.wait, which returns
// when that kernel has completed and its writes are visible.
template <class... KArgs, class... Args>
int launch_overlapped(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr; cfg.numAttrs = 1;
    KVC_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...));
    return KVC_OK;
}

int check_cache(const kvc_cache *c, const char *who, bool is_k) {
    KVC_REQUIRE(c && c->encoded && c->block_info && c->thread_info && c->book && c->q.min_int && c->q.scale,
                "%s: null pointer in the %s cache", who, is_k ? "K" : "V");
    KVC_REQUIRE(c->q.min_bytes == 1 || c->q.min_bytes == 2, "%s: min_bytes must be 1 or 2", who);
    KVC_REQUIRE(c->q.tok_div > 0, "%s: tok_div must be positive", who);
    KVC_REQUIRE((reinterpret_cast<uintptr_t>(c->book) & 15) == 0 && (reinterpret_cast<uintptr_t>(c->block_info) & 7) == 0,
                "%s: book must be 16-byte and block_info 8-byte aligned", who);
    if (is_k) {
        KVC_REQUIRE(c->q.sc == 0 || c->q.tok_div % 64 == 0,
                    "%s: K units that depend on the channel must cover whole 64-token blocks", who);
        // the kernels fetch the units of 4 neighbouring channels with one load
        KVC_REQUIRE(c->q.sc == 0 || (c->q.sc == 1 && c->q.sj % 4 == 0 && c->q.sb % 4 == 0 && c->q.sh % 4 == 0 &&
                                     (reinterpret_cast<uintptr_t>(c->q.scale) & 7) == 0 &&
                                     (reinterpret_cast<uintptr_t>(c->q.min_int) & (c->q.min_bytes == 1 ? 3 : 7)) == 0),
                    "%s: per-channel K units must be contiguous over the channels and 8-byte aligned", who);
    }
    else KVC_REQUIRE(c->q.sc == 0, "%s: V units that depend on the channel are not supported by the fused kernels", who);
    return KVC_OK;
}

// the query heads of a KV head are processed in chunks of 4, 2 or 1 by the two unfused kernels
int next_chunk(long long remaining) { return remaining >= 4 ? 4 : (remaining >= 2 ? 2 : 1); }

}  // namespace

extern "C" int kvc_fused_qk(const kvc_cache *k, int64_t T, int64_t B, int64_t Hkv, int64_t Hq,
                            const void *q, void *out, int out_f32, int32_t *status, kvc_stream_t stream) {
    if (int rc = check_cache(k, "kvc_fused_qk", true)) return rc;
    KVC_REQUIRE(q && out && status, "kvc_fused_qk: null pointer");
    KVC_REQUIRE(B > 0 && Hkv > 0 && Hq > 0 && Hq % Hkv == 0 && T >= 0 && T % 64 == 0, "kvc_fused_qk: bad shape");
    KVC_REQUIRE(B * Hkv <= 65535, "kvc_fused_qk: B*Hkv exceeds the grid limit");
    if (T == 0) return KVC_OK;
    const CacheDev kc = to_dev(*k);
    const dim3 grid((unsigned)((T + 255) / 256), (unsigned)(B * Hkv));
    const long long Gt = Hq / Hkv;
    for (long long g0 = 0; g0 < Gt;) {
        const int G = next_chunk(Gt - g0);
#define KVC_QK(GG)                                                                                              \
    {                                                                                                           \
        static kvc_launch_slot slot;                                                                            \
        int occ = 0;                                                                                            \
        const size_t smem = unfused_smem<QkSmem<GG>>(kc);                                                       \
        if (int rc = kvc_prepare(slot, reinterpret_cast<const void *>(fused_qk_kernel<GG>), NTHR, smem, &occ)) return rc; \
        fused_qk_kernel<GG><<<grid, NTHR, smem, kvc_cu(stream)>>>(                                \
            kc, T, B, Hkv, Hq, g0, reinterpret_cast<const __half *>(q), out, out_f32, status);                  \
    }
        if (G == 4) KVC_QK(4) else if (G == 2) KVC_QK(2) else KVC_QK(1)
#undef KVC_QK
        g0 += G;
    }
    KVC_LAUNCH_OK();
    return KVC_OK;
}

extern "C" int kvc_fused_pv(const kvc_cache *v, int64_t T, int64_t B, int64_t Hkv, int64_t Hq,
                            const void *P, void *out, int32_t *status, kvc_stream_t stream) {
    if (int rc = check_cache(v, "kvc_fused_pv", false)) return rc;
    KVC_REQUIRE(P && out && status, "kvc_fused_pv: null pointer");
    KVC_REQUIRE(B > 0 && Hkv > 0 && Hq > 0 && Hq % Hkv == 0 && T >= 0 && T % 128 == 0, "kvc_fused_pv: bad shape");
    KVC_REQUIRE(B * Hkv <= 65535, "kvc_fused_pv: B*Hkv exceeds the grid limit");
    if (T == 0) return KVC_OK;
    const CacheDev vc = to_dev(*v);
    const dim3 grid((unsigned)((T + 255) / 256), (unsigned)(B * Hkv));
    const long long Gt = Hq / Hkv;
    for (long long g0 = 0; g0 < Gt;) {
        const int G = next_chunk(Gt - g0);
#define KVC_PV(GG)                                                                                              \
    {                                                                                                           \
        static kvc_launch_slot slot;                                                                            \
        int occ = 0;                                                                                            \
        const size_t smem = unfused_smem<PvSmem<GG>>(vc);                                                       \
        if (int rc = kvc_prepare(slot, reinterpret_cast<const void *>(fused_pv_kernel<GG>), NTHR, smem, &occ)) return rc; \
        fused_pv_kernel<GG><<<grid, NTHR, smem, kvc_cu(stream)>>>(                                \
            vc, T, B, Hkv, Hq, g0, reinterpret_cast<const __half *>(P), reinterpret_cast<__half *>(out), status); \
    }
        if (G == 4) KVC_PV(4) else if (G == 2) KVC_PV(2) else KVC_PV(1)
#undef KVC_PV
        g0 += G;
    }
    KVC_LAUNCH_OK();
    return KVC_OK;
}

namespace {
// The sum over a head's partial outputs: CTA = (sequence, query head); a warp takes every eighth row, 4 channels a lane, 8 rows on their way at
// once.  Bound by the trips to L2.  (As a reduction and a conversion of torch's, 128 groups of 32 heads: 5.5 and 2.0 us and a launch more; now 3.0.)
__global__ void __launch_bounds__(256) pv_sum_kernel(const __half *__restrict__ part, long long groups, long long rows, __half *__restrict__ out) {
    __shared__ float4 sums[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const __half *src = part + (long long)blockIdx.x * 128 + lane * 4;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
    for (long long g0 = warp; g0 < groups; g0 += 64) {
        uint2 x[8];
#pragma unroll
        for (int k = 0; k < 8; k++) if (g0 + 8 * k < groups) x[k] = __ldg(reinterpret_cast<const uint2 *>(src + (g0 + 8 * k) * rows * 128));
#pragma unroll
        for (int k = 0; k < 8; k++) if (g0 + 8 * k < groups) {
            const float2 lo = __half22float2(*reinterpret_cast<const __half2 *>(&x[k].x)), hi = __half22float2(*reinterpret_cast<const __half2 *>(&x[k].y));
            a.x += lo.x; a.y += lo.y; a.z += hi.x; a.w += hi.y;
        }
    }
    sums[warp][lane] = a;
    __syncthreads();
    if (warp) return;
#pragma unroll
    for (int w = 1; w < 8; w++) { const float4 o = sums[w][lane]; a.x += o.x; a.y += o.y; a.z += o.z; a.w += o.w; }
    __half2 r[2] = {__floats2half2_rn(a.x, a.y), __floats2half2_rn(a.z, a.w)};
    *reinterpret_cast<uint2 *>(out + (long long)blockIdx.x * 128 + lane * 4) = *reinterpret_cast<const uint2 *>(r);
}
}  // namespace

extern "C" int kvc_pv_sum(const void *part, int64_t groups, int64_t B, int64_t Hq, void *out, kvc_stream_t stream) {
    KVC_REQUIRE(part && out, "kvc_pv_sum: null pointer");
    KVC_REQUIRE(groups > 0 && B > 0 && Hq > 0 && B * Hq < (1ll << 31), "kvc_pv_sum: bad shape");
    KVC_REQUIRE(((reinterpret_cast<uintptr_t>(part) | reinterpret_cast<uintptr_t>(out)) & 7) == 0, "kvc_pv_sum: part and out must be 8-byte aligned");
    pv_sum_kernel<<<(unsigned)(B * Hq), 256, 0, kvc_cu(stream)>>>(reinterpret_cast<const __half *>(part), groups, B * Hq, reinterpret_cast<__half *>(out));
    KVC_LAUNCH_OK();
    return KVC_OK;
}

// Diagnostics for tests of the bounded waits (kvc_attn_debug): process-wide, read at every launch.
static int g_wait_limit = 0, g_starve = 0;
extern "C" void kvc_attn_debug(int wait_limit, int starve) { g_wait_limit = wait_limit; g_starve = starve; }

// What a workspace is sized for: runs of 256-token tiles for this many takers per SM (kvc_attn_splits); the kernels' plans may
// cut twice as many.
constexpr int ATTN_CTAS_PER_SM = 3;
// items a resident CTA should get on average: enough that the draws even out the CTAs' speeds and the
// last items end close together, few enough that the per-item work (q, partial results) stays small
constexpr int ATTN_ITEMS_PER_CTA = 4;

template <int G, bool BULK, bool TEAM> auto attn_kernel() {
    if constexpr (G == 1) return attn_one_kernel<BULK, TEAM>;
    else return attn_rows_kernel<G, BULK, TEAM>;
}
template <int G> size_t attn_smem(const AttnParams &p, int workers) {
    if constexpr (G == 1) return one_smem(p, workers);
    else return rows_smem<G>(p, workers);
}

// How the columns are cut when the caller leaves it to the library: long runs of `tps` tiles, and at the
// end of every column short runs of half that, enough of them that each resident CTA finds about two
// short items to finish with.  The short items are handed out last (the item order puts them behind
// all long ones), so the CTAs of a launch end within one short item of each other.
struct RunPlan { int tps, long_runs, short_tiles, splits; };
static RunPlan plan_runs(long long n_tiles, long long cols, long long P) {      // P: CTAs (grouped queries: workers) at work
    RunPlan r = {1, 1, 1, 1};
    if (n_tiles <= 0 || cols <= 0) { r.tps = 0; r.long_runs = 1; r.short_tiles = 0; return r; }
    long long tps = cols * n_tiles / (P * ATTN_ITEMS_PER_CTA);       // tiles per long item
    if (tps < 1) tps = 1;
    if (tps > n_tiles) tps = n_tiles;
    // (items of a single tile pay the per-item work too often: measured slower than no short runs at all)
    long long short_tiles = tps >= 4 ? tps / 2 : tps;
    long long short_region = 0;                                      // tiles of a column cut into short runs
    if (short_tiles < tps) {
        short_region = (2 * P * short_tiles + cols - 1) / cols;       // about two short items per CTA over all columns
        short_region = (short_region + tps - 1) / tps * tps;
        if (short_region > n_tiles) short_region = n_tiles;
    }
    long long long_runs = (n_tiles - short_region) / tps;
    short_region = n_tiles - long_runs * tps;
    const long long short_runs = (short_region + short_tiles - 1) / short_tiles;
    r.tps = (int)tps; r.long_runs = (int)long_runs; r.short_tiles = (int)short_tiles; r.splits = (int)(long_runs + short_runs);
    return r;
}

extern "C" int kvc_attn_splits(int64_t T, int64_t B, int64_t Hkv, int sm_count) {
    if (T <= 0 || B <= 0 || Hkv <= 0) return 1;
    if (sm_count <= 0) sm_count = kvc_sm_count();
    return plan_runs((T + 255) / 256, B * Hkv, (long long)ATTN_CTAS_PER_SM * sm_count).splits;
}

// bytes of the zero-initialised head of a workspace: the two scheduling counters
constexpr int64_t ATTN_COUNTER_BYTES = 256;

extern "C" int64_t kvc_attn_workspace(int64_t B, int64_t Hq, int splits) {
    if (splits < 1) splits = 1;
    return ATTN_COUNTER_BYTES + B * Hq * (int64_t)(splits > 1 ? splits : 1) * ATTN_PART_FLOATS * 4;    // one run still leaves a partial result when a tail follows
}

extern "C" int kvc_attn_decode(const kvc_cache *k, const kvc_cache *v, int64_t T, int64_t B, int64_t Hkv, int64_t Hq,
                               const void *q, float scaling, const void *ktail, const void *vtail, int64_t Tr,
                               void *out, int splits, void *workspace, int64_t workspace_bytes,
                               int32_t *status, kvc_stream_t stream) {
    if (T > 0) {      // with nothing compressed yet only the fp16 tail is read and the caches may be NULL
        if (int rc = check_cache(k, "kvc_attn_decode", true)) return rc;
        if (int rc = check_cache(v, "kvc_attn_decode", false)) return rc;
    }
    KVC_REQUIRE(q && out && status, "kvc_attn_decode: null pointer");
    KVC_REQUIRE(B > 0 && Hkv > 0 && Hq > 0 && Hq % Hkv == 0, "kvc_attn_decode: bad head counts");
    KVC_REQUIRE(T >= 0 && T % 128 == 0, "kvc_attn_decode: the compressed length must be a multiple of 128, got %lld", (long long)T);
    KVC_REQUIRE(Tr >= 0 && (Tr == 0 || (ktail && vtail)), "kvc_attn_decode: tail pointers missing");
    KVC_REQUIRE(T + Tr > 0, "kvc_attn_decode: empty cache");
    KVC_REQUIRE(Tr == 0 || ((reinterpret_cast<uintptr_t>(ktail) & 15) == 0), "kvc_attn_decode: ktail must be 16-byte aligned");
    const long long n_tiles = (T + 255) / 256, cols = B * Hkv;
    KVC_REQUIRE(T < (1ll << 31) - 1024 && cols < (1ll << 30) && B * Hq < (1ll << 30), "kvc_attn_decode: shape too large");
    // every column is cut into runs of tiles; each (column, run) is one item of work.  splits > 0: that many
    // equal runs.  Otherwise long runs and, at the end of each column, short ones (plan_runs).
    int tps, long_runs, short_tiles;
    const int asked = splits;
    if (splits <= 0) {
        const RunPlan r = plan_runs(n_tiles, cols, (long long)ATTN_CTAS_PER_SM * kvc_sm_count());
        tps = r.tps; long_runs = r.long_runs; short_tiles = r.short_tiles; splits = r.splits;
    } else {
        if (splits > n_tiles) splits = (int)(n_tiles > 0 ? n_tiles : 1);
        tps = (int)((n_tiles + splits - 1) / splits);
        splits = tps > 0 ? (int)((n_tiles + tps - 1) / tps) : 1;
        long_runs = splits; short_tiles = tps;
    }
    KVC_REQUIRE(cols * splits < (1ll << 31) - (1ll << 20), "kvc_attn_decode: too many items");
    if (splits > 1) {
        KVC_REQUIRE(workspace && workspace_bytes >= kvc_attn_workspace(B, Hq, splits),
                    "kvc_attn_decode: workspace needs %lld bytes for %d splits", (long long)kvc_attn_workspace(B, Hq, splits), splits);
        KVC_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 15) == 0, "kvc_attn_decode: workspace must be 16-byte aligned");
    }
    AttnParams p;
    if (T > 0) { p.k = to_dev(*k); p.v = to_dev(*v); }
    else { p.k = CacheDev(); p.v = CacheDev(); p.k.q.tok_div = p.v.q.tok_div = 1; }
    p.T = T; p.B = B; p.Hkv = Hkv; p.Hq = Hq; p.Tr = Tr;
    p.q = reinterpret_cast<const __half *>(q);
    p.ktail = reinterpret_cast<const __half *>(ktail); p.vtail = reinterpret_cast<const __half *>(vtail);
    p.out = reinterpret_cast<__half *>(out);
    p.scaling = scaling; p.splits = splits; p.tiles_per_split = tps; p.long_runs = long_runs; p.short_tiles = short_tiles;
    p.n_tiles = (int)n_tiles;
    p.team = p.brief = p.spare = 0;
    p.work = cols * splits;
    // with a workspace the CTAs draw their items from its counters (zero before the first launch, left zeroed)
    const bool have_ws = workspace && workspace_bytes >= ATTN_COUNTER_BYTES && (reinterpret_cast<uintptr_t>(workspace) & 15) == 0;
    p.sched = have_ws ? reinterpret_cast<int *>(workspace) : nullptr;
    p.ws_part = have_ws ? reinterpret_cast<float *>(reinterpret_cast<uint8_t *>(workspace) + ATTN_COUNTER_BYTES) : nullptr;
    // The tail belongs to the merge kernel whenever the attention kernel can leave partial results for it (a
    // workspace with room for them) or has nothing to do at all (no compressed part); only a caller without a
    // workspace gets the tail from the attention kernel itself.
    const bool ws_parts = have_ws && workspace_bytes >= kvc_attn_workspace(B, Hq, splits);
    const bool tail_in_merge = Tr > 0 && (T == 0 || splits > 1 || ws_parts);
    p.partial = splits > 1 || (tail_in_merge && T > 0);
    p.status = status;
    p.wait_limit = g_wait_limit > 0 ? g_wait_limit : KVC_WAIT_LIMIT;
    p.starve = g_starve;
    p.slotK_bytes = slot_bytes_of(p.k.max_block);
    p.slotV_bytes = slot_bytes_of(p.v.max_block);
    // bulk copies widen every block to 16-byte boundaries: both streams must start on one
    const bool bulk = T > 0 && (reinterpret_cast<uintptr_t>(k->encoded) & 15) == 0 && (reinterpret_cast<uintptr_t>(v->encoded) & 15) == 0;
    const int sms = kvc_sm_count();
    const long long Gt = Hq / Hkv;
    long long attn_ctas = 0;
    if (T > 0) {
        // The kernels count in steps of 128 tokens.  The workspace, sized for `splits` runs of 256-token tiles, holds twice as many
        // of their partial results: with many small workers the items are finer where it may be so.
        p.n_tiles = (int)(T / 128);
        p.tiles_per_split *= 2; p.short_tiles *= 2;
        const int heads = (int)((Gt + (Gt + 7) / 8 - 1) / ((Gt + 7) / 8));                   // of the first launch
        const long long most = (long long)rows_fit(p, heads) * sms;                         // workers of a full device
        if (p.partial && ws_parts) {
            RunPlan r = {0, 0, 0, 0};
            // (with grouped queries the plan counts five workers per SM also where the launch has fewer: the items are finer for it.  8 heads, four
            // workers: 16 x 8 columns of 16384 tokens 338 us, with a plan for four 345; 32 x 2 columns 191 and 195; 16 x 8 of 4096 115 either way.  Three
            // workers, as the stream's largest block is unknown: 399 and 402 us.)
            if (asked <= 0) r = plan_runs(p.n_tiles, cols, heads == 1 ? most : (long long)ROWS_PLANNED * sms);
            // The caller's runs in halves where that is fewer steps one after the other: a worker takes a run's steps in turn, each
            // with 128 threads.  (32 columns, 2 heads each, 2048 tokens in 4
            // runs: 37.0 us, in halves 22.1; 64 columns in 8 runs: 29.4, in halves 31.3, as the halves no longer go in one round.)
            else if ((2 * cols * splits + most - 1) / most < 2 * ((cols * splits + most - 1) / most)) {
                r.tps = r.short_tiles = tps;
                r.splits = r.long_runs = (p.n_tiles + tps - 1) / tps;
            }
            if (r.splits > 0 && r.splits <= 2 * splits && cols * r.splits < (1ll << 31) - (1ll << 20)) {
                p.tiles_per_split = r.tps; p.long_runs = r.long_runs; p.short_tiles = r.short_tiles; splits = p.splits = r.splits;
            }
        }
        p.work = cols * splits;
        for (long long g0 = 0; g0 < Gt; g0 += p.nh) {
            // Heads per launch: every launch decodes the whole cache, so up to 8 go together, in launches of equal shares.
            // (32 sequences x 16384 tokens, 2 x 8 heads, K rel 0.05: 321 us in two launches of 4, 181 us in one.)
            const long long launches = (Gt - g0 + 7) / 8;
            p.g0 = g0; p.nh = (int)((Gt - g0 + launches - 1) / launches);
#define KVC_AT(GG)                                                                                              \
    {                                                                                                           \
        p.brief = p.spare = 0;                                                                                  \
        int workers = rows_fit(p, GG);                                                                          \
        /* (with a tail and columns for all workers a pass of the tail is no step: 1023 columns of 2048 tokens and 64 rows, 4 heads, */ \
        /* a worker per column 440 us, teams as chosen for 18 steps 503) */                                     \
        p.team = p.partial || (Tr > 0 && cols >= (long long)workers * sms) ? 0 : rows_team(cols, p.n_tiles + (Tr + 127) / 128, workers, sms); \
        if (p.team) workers = p.team * (int)spread(cols, workers / p.team, sms).per_sm;                         \
        /* (short runs at the end of the columns fill the last round up; a single round spreads over all SMs) */ \
        else if (const Spread s = spread(p.work, workers, sms); p.long_runs == splits || s.rounds == 1) workers = (int)s.per_sm; \
        /* (steps that a worker takes one after the other) */                                                   \
        const long long steps = p.team ? spread(cols, workers / p.team, sms).rounds * ((p.n_tiles + p.team - 1) / p.team) \
                                       : spread(p.work, workers, sms).rounds * std::min(p.tiles_per_split, p.n_tiles);     \
        p.brief = GG > 1 && steps <= BRIEF_STEPS;                                                               \
        if (p.brief && attn_smem<GG>(p, workers) > MAX_CTA_SHARED) p.brief = 0;                                 \
        p.spare = GG > 1 && !p.brief && attn_smem<GG>(p, workers) + 4 * KVC_LUT_SIZE <= MAX_CTA_SHARED;         \
        const size_t smem = attn_smem<GG>(p, workers);                                                          \
        p.workers = workers;                                                                                    \
        /* (one head) Without a tail the merge kernel has nothing to do beside the last items, and a CTA of more than four workers leaves it no room there: let go early it */ \
        /* made long launches slower than one that is let go by a worker's end.  (Kernels by other ones, in a graph, let go early and now: 4 columns of 32768 tokens 27.2 and 25.8 us, of */ \
        /* 65536 47.4 and 45.9, 16 of 20480 49.1 and 48.4, 8 of 65536 76.8 and 74.8; one behind the other 24.2 and 24.8, 45.3 and 42.6, 46.5 and 45.0, 74.4 and 71.4; 256 of */ \
        /* 4096 120.6 and 120.8.  With up to four workers, let go early and late: 32 of 256 7.9 and 10.8, 16 of 4096 13.8 and 14.1.) */ \
        p.early = Tr > 0 || workers <= 4;                                                                       \
        /* (threads that only help to load the tables would take the merge kernel's place beside a brief launch) */ \
        const int threads = 128 * (GG == 1 || p.brief ? workers : rows_workers<GG>());                           \
        static kvc_launch_slot slots[4];                                                                        \
        auto *kernel = p.team ? (bulk ? attn_kernel<GG, true, true>() : attn_kernel<GG, false, true>())         \
                              : (bulk ? attn_kernel<GG, true, false>() : attn_kernel<GG, false, false>());      \
        int occ = 0;                                                                                            \
        if (int rc = kvc_prepare(slots[2 * (p.team != 0) + bulk], reinterpret_cast<const void *>(kernel), threads, smem, &occ)) return rc; \
        KVC_REQUIRE(occ >= 1, "kvc_attn_decode: %zu bytes of shared memory do not fit an SM", smem);             \
        long long ctas = p.team ? p.work : (p.work + workers - 1) / workers;                                    \
        if (ctas > sms) ctas = sms;                                                                             \
        attn_ctas = ctas;                                                                                       \
        if (int rc = launch_overlapped(kernel, dim3((unsigned)ctas), dim3(threads), smem, kvc_cu(stream), p)) return rc; \
    }
            if (p.nh > 4) KVC_AT(8) else if (p.nh > 2) KVC_AT(4) else if (p.nh > 1) KVC_AT(2) else KVC_AT(1)
#undef KVC_AT
        }
    }
    if (p.partial || tail_in_merge) {
        TailArgs ta = {};
        if (tail_in_merge) {
            ta.q = p.q; ta.ktail = p.ktail; ta.vtail = p.vtail; ta.Tr = Tr;
            ta.B = (int)B; ta.Hkv = (int)Hkv; ta.Hq = (int)Hq; ta.scaling = scaling;
        }
        const bool pairs = (reinterpret_cast<uintptr_t>(ta.vtail) & 3) == 0, apart = B * Hq <= 2 * (sms - attn_ctas);
        auto *merge = apart ? (pairs ? attn_merge_kernel<true, 128> : attn_merge_kernel<false, 128>) : (pairs ? attn_merge_kernel<true, 96> : attn_merge_kernel<false, 96>);
        if (int rc = launch_overlapped(merge, dim3((unsigned)(B * Hq)), dim3(MERGE_THREADS), 0, kvc_cu(stream),
                                       (const float *)p.ws_part, p.out, T > 0 ? splits : 0, ta)) return rc;
    }
    KVC_LAUNCH_OK();
    return KVC_OK;
}

extern "C" int kvc_attn_decode_packed(const kvc_attn_args *args, kvc_stream_t stream) {
    KVC_REQUIRE(args, "kvc_attn_decode_packed: null pointer");
    kvc_attn_args a;
    memcpy(&a, args, sizeof(a));                            // (wherever the caller packed them)
    return kvc_attn_decode(a.T > 0 ? &a.k : nullptr, a.T > 0 ? &a.v : nullptr, a.T, a.B, a.Hkv, a.Hq, a.q, a.scaling, a.ktail, a.vtail,
                           a.Tr, a.out, a.splits, a.workspace, a.workspace_bytes, a.status, stream);
}

// ---- decode attention for callers that cannot allocate device memory ------------------------------
// Some hosts of this library may not call cudaMalloc at all: an inference server whose memory pool
// owns every byte of the device and forbids side allocations, a plugin loaded into a process that
// runs under a fixed memory budget, or code that runs where an allocation would synchronise the
// device at the wrong moment.  For them the split-KV scratch of the attention kernel (per-head
// counters and the per-split partial results) lives in this fixed array instead of a workspace the
// caller has to provide.  Every context that loads the library holds these bytes until it ends.
#define KVC_STATIC_SCRATCH_BYTES (4 << 20)
static __device__ __align__(256) unsigned char g_attn_scratch[KVC_STATIC_SCRATCH_BYTES];

namespace {
std::atomic<void *> g_scratch_ptr[KVC_MAX_CONTEXTS];

// The array's name is only a host-side handle in host code; the device address has to be asked for, once per context,
// with that context current (each has an array of its own).
int static_scratch(void **ptr) {
    const int ctx = kvc_context();
    *ptr = ctx >= 0 ? g_scratch_ptr[ctx].load(std::memory_order_relaxed) : nullptr;
    if (*ptr) return KVC_OK;
    KVC_CUDA_OK(cudaGetSymbolAddress(ptr, g_attn_scratch));
    if (ctx >= 0) g_scratch_ptr[ctx].store(*ptr, std::memory_order_relaxed);
    return KVC_OK;
}
}  // namespace

extern "C" int64_t kvc_attn_static_capacity(void) { return KVC_STATIC_SCRATCH_BYTES; }

extern "C" int kvc_attn_decode_static(const kvc_cache *k, const kvc_cache *v, int64_t T, int64_t B, int64_t Hkv, int64_t Hq,
                                      const void *q, float scaling, const void *ktail, const void *vtail, int64_t Tr,
                                      void *out, int splits, int32_t *status, kvc_stream_t stream) {
    KVC_REQUIRE(B > 0 && Hkv > 0 && Hq > 0 && T >= 0, "kvc_attn_decode_static: bad shape");
    // partial results per head: kvc_attn_decode never cuts a column into more runs than it has tiles
    const long long n_tiles = (T + 255) / 256;
    const int parts = splits <= 0 ? kvc_attn_splits(T, B, Hkv, 0) : (int)(splits > n_tiles ? (n_tiles > 0 ? n_tiles : 1) : splits);
    const int64_t need = kvc_attn_workspace(B, Hq, parts);
    if (need > KVC_STATIC_SCRATCH_BYTES) {
        kvc_set_error("kvc_attn_decode_static: B=%lld x Hq=%lld x %d splits needs %lld bytes of scratch, the built-in "
                      "array holds %d; lower `splits` or use kvc_attn_decode with a workspace",
                      (long long)B, (long long)Hq, parts, (long long)need, KVC_STATIC_SCRATCH_BYTES);
        return KVC_ERR_CAPACITY;
    }
    void *scratch = nullptr;
    if (int rc = static_scratch(&scratch)) return rc;
    // the array keeps whatever the previous call left: the scheduling counters must start at zero
    KVC_CUDA_OK(cudaMemsetAsync(scratch, 0, ATTN_COUNTER_BYTES, kvc_cu(stream)));
    return kvc_attn_decode(k, v, T, B, Hkv, Hq, q, scaling, ktail, vtail, Tr, out, splits, scratch, need, status, stream);
}
