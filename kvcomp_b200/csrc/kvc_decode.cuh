// Per-thread Huffman vector decoder shared by the plain decoder and the fused attention kernels,
// and the helpers that stage compressed blocks in shared memory.
//
// A vector is 128 symbols, MSB-first, starting on a byte boundary (kernels.cu:237-291 walks it
// one bit at a time through a tree in global memory).  Here the block's bytes sit in shared
// memory, the thread keeps 64 bits of the stream in two registers and looks up KVC_LUT_BITS
// bits at a time in a shared-memory table that returns up to three symbols per lookup; codes
// longer than the window continue bit by bit from the tree node the window leads to.
#pragma once

#include "kvc_common.cuh"

#define KVC_DECODE_OVERRUN 6              // positions past 127 a decoder may emit (two lookups per round)

struct KvcBookSmem {                      // per-CTA copy of the decode structures of one book
    uint32_t tree[512];
    uint32_t lut[KVC_LUT_SIZE];
};

// The decode table as the loop below wants it: a book's entries {(symbols << 6) | bits, s0, s1, s2} with 16 - bits in place
// of the bits (an entry without a complete code: no symbols, still told by bits 6-7).
__device__ __forceinline__ void kvc_load_lut(uint32_t *lut, const void *book, int tid, int nthr) {
    const uint4 *src = reinterpret_cast<const uint4 *>(reinterpret_cast<const uint8_t *>(book) + KVC_BOOK_OFF_LUT);
    auto form = [](uint32_t e) { return e + 16u - 2u * (e & 63u); };
    for (int i = tid; i < KVC_LUT_SIZE / 4; i += nthr) {
        const uint4 e = src[i];
        reinterpret_cast<uint4 *>(lut)[i] = make_uint4(form(e.x), form(e.y), form(e.z), form(e.w));
    }
}
// Two books' tables, up to four entries of 16 bytes of each on their way at once: a launch of few threads otherwise waits for one
// after the other (two workers of 128 threads: eight trips to L2).  (Attention, a pass among others: 12 columns of 2816 tokens, 6 heads, 22.2 and 21.7 us; 256
// columns of 4096, one head, 128.5 and 128.2.)
__device__ __forceinline__ void kvc_load_luts(uint32_t *lut0, uint32_t *lut1, const void *book0, const void *book1, int tid, int nthr) {
    const uint4 *src0 = reinterpret_cast<const uint4 *>(reinterpret_cast<const uint8_t *>(book0) + KVC_BOOK_OFF_LUT);
    const uint4 *src1 = reinterpret_cast<const uint4 *>(reinterpret_cast<const uint8_t *>(book1) + KVC_BOOK_OFF_LUT);
    constexpr int N = KVC_LUT_SIZE / 4, AHEAD = 4;
    auto form = [](const uint4 &e) { return make_uint4(e.x + 16u - 2u * (e.x & 63u), e.y + 16u - 2u * (e.y & 63u), e.z + 16u - 2u * (e.z & 63u), e.w + 16u - 2u * (e.w & 63u)); };
    for (int i = tid; i < N; i += AHEAD * nthr) {
        uint4 a[AHEAD], b[AHEAD];
#pragma unroll
        for (int j = 0; j < AHEAD; j++) if (i + j * nthr < N) { a[j] = __ldg(src0 + i + j * nthr); b[j] = __ldg(src1 + i + j * nthr); }
#pragma unroll
        for (int j = 0; j < AHEAD; j++) if (i + j * nthr < N) {
            reinterpret_cast<uint4 *>(lut0)[i + j * nthr] = form(a[j]);
            reinterpret_cast<uint4 *>(lut1)[i + j * nthr] = form(b[j]);
        }
    }
}
__device__ __forceinline__ void kvc_load_book(KvcBookSmem &b, const void *book, int tid, int nthr) {
    const uint4 *src = reinterpret_cast<const uint4 *>(reinterpret_cast<const uint8_t *>(book) + KVC_BOOK_OFF_TREE);
    for (int i = tid; i < 512 / 4; i += nthr) reinterpret_cast<uint4 *>(b.tree)[i] = src[i];
    kvc_load_lut(b.lut, book, tid, nthr);
}

// the wide decode tree, read only for codes longer than the table's window
struct KvcTreeShared {
    uint32_t addr;
    __device__ __forceinline__ uint32_t operator()(uint32_t node) const;
};
struct KvcTreeGlobal {                    // for kernels short of shared memory
    const uint32_t *nodes;
    __device__ __forceinline__ KvcTreeGlobal(const void *book) : nodes(reinterpret_cast<const uint32_t *>(reinterpret_cast<const uint8_t *>(book) + KVC_BOOK_OFF_TREE)) {}
    __device__ __forceinline__ uint32_t operator()(uint32_t node) const { return nodes[node]; }
};

// Copy the bytes [off, off+n) of `encoded` into `slot` so that slot and source agree modulo 16:
// the first stream byte lands at slot[lead], lead = address & 15.  Whole 16-byte chunks inside the
// buffer move as 128-bit loads; the ragged edges move bytewise, never touching memory outside
// [encoded, encoded + encoded_bytes).  Returns lead.  All `nthr` threads of the group take part.
__device__ __forceinline__ uint32_t kvc_stage_block(uint8_t *slot, const uint8_t *__restrict__ encoded,
                                                    long long encoded_bytes, long long off, uint32_t n,
                                                    int tid, int nthr) {
    const uint8_t *src = encoded + off;
    const uint32_t lead = (uint32_t)(reinterpret_cast<uintptr_t>(src) & 15);
    const uint8_t *a0 = src - lead;                                  // 16-byte aligned
    const uint32_t chunks = (lead + n + 15) >> 4;
    const uint8_t *lo = encoded, *hi = encoded + encoded_bytes;
    for (uint32_t c = tid; c < chunks; c += nthr) {
        const uint8_t *p = a0 + 16 * c;
        if (p >= lo && p + 16 <= hi) {
            *reinterpret_cast<uint4 *>(slot + 16 * c) = *reinterpret_cast<const uint4 *>(p);
        } else {
            for (int k = 0; k < 16; k++) slot[16 * c + k] = (p + k >= lo && p + k < hi) ? p[k] : (uint8_t)0;
        }
    }
    return lead;
}

// ---- bulk asynchronous copies (TMA, untiled) completing on a shared-memory mbarrier -------------
__device__ __forceinline__ uint32_t kvc_smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void kvc_mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(kvc_smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void kvc_mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void kvc_mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(kvc_smem_addr(bar)), "r"(bytes) : "memory");
}
// src and dst 16-byte aligned, bytes a multiple of 16 and > 0
__device__ __forceinline__ void kvc_bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(kvc_smem_addr(dst)), "l"(src), "r"(bytes), "r"(kvc_smem_addr(bar)) : "memory");
}
// Bounded wait for the phase with the given parity: at most `limit` tries.  Returns false if the phase
// never completed.
#define KVC_WAIT_LIMIT (1 << 22)
__device__ __forceinline__ bool kvc_mbar_wait(uint64_t *bar, uint32_t parity, int limit = KVC_WAIT_LIMIT) {
    const uint32_t a = kvc_smem_addr(bar);
    for (int it = 0; it < limit; it++) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done) : "r"(a), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}

__device__ __forceinline__ int kvc_dp4a_us(uint32_t a_u8x4, uint32_t b_s8x4, int c) {
    int d;
    asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a_u8x4), "r"(b_s8x4), "r"(c));
    return d;
}
__device__ __forceinline__ int kvc_dp4a_uu(uint32_t a_u8x4, uint32_t b_u8x4, int c) {
    int d;
    asm("dp4a.u32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a_u8x4), "r"(b_u8x4), "r"(c));
    return d;
}

__device__ __forceinline__ uint32_t kvc_lds32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t KvcTreeShared::operator()(uint32_t node) const { return kvc_lds32(addr + node * 4); }
__device__ __forceinline__ uint2 kvc_lds64(uint32_t addr) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}

// Whether the decoder has to test every table entry for "no code ends in this window": books with a
// code longer than the window, and books whose code is not complete (a single symbol, or a tree taken
// from a caller's tensor with a missing branch): a corrupt stream can then show bit patterns that
// belong to no code, and the escape-free loop would not advance on them.
__device__ __forceinline__ bool kvc_book_needs_escape(const void *book) {
    return reinterpret_cast<const kvc_book_header *>(book)->escape != 0;    // set for a code beyond the window too
}

// Decode one vector.  slot_s: shared-space address of the staged block (16-byte aligned; the word before it is readable);
// byte_pos: where the vector starts in it; lut_s: shared-space address of the book's table (kvc_load_lut's form); tree: its
// tree (KvcTree*).
// The stream's next bits lie in the register pair (hi, lo), `off` bits from its top; the decoder state is (position << 6) | f
// with f = 34 - off, kept in 0..31: `(hi, lo) >> f` then has the next 30 bits below bit 30, the first window's table offset is
// one shift and one mask away, and the second one's too, as a table entry's low five bits are the shift (16 - bits consumed)
// that brings the bits behind it to the same place.  Both windows of a round lie in that one word, so nothing is chosen in between
// and the chain from one lookup to the next is a shift and a mask.  Applying an entry is one add of its low byte; the two
// 16s of a round are the 32 that a refill (or clearing bit 5) takes off again.
// (What bounds a decode loop is issue and the shared-memory pipe together with the chain of lookups.  With the second window cut
// from words chosen by the state, one more shift per window and an end test per round: attention over 16 x 32768 tokens, 8 x 4
// heads, 724 us, now 652; one head, 8 x 4096 tokens, 142 and 135.)
// emit(e, a, s0, s1): `e` holds up to three symbols in bytes 1..3 for positions c..c+2 of the vector (unused
// bytes are 0; byte 0 is the table entry's advance byte: its bits 6-7 count the symbols); a = (base + c) << SHIFT:
// the position counter starts at `base`, so a consumer that keeps one record of 2^SHIFT bytes per
// position at shared address A passes base = A >> SHIFT and gets the record's address with no add;
// s0, s1: the state before and after the lookup (position from bit 6 up), for consumers that track word borders.
// The end of the vector is tested once per two lookups, so emit may be handed symbols for positions up to
// 127 + KVC_DECODE_OVERRUN; the consumer keeps room for them (zero weights, padding).
// ESC = false is for books whose longest code fits the table window: no escape test in the loop.
// Every round advances by at least one symbol, so the loop ends after at most 128 rounds; a corrupt
// stream can read at most a few hundred bytes past its vector, for which the kernels keep padding
// behind the last slot.  Returns false when the bits do not form valid codes.
template <bool ESC, int SHIFT, class Emit, class Tree = KvcTreeShared>
__device__ __forceinline__ bool kvc_decode_vector(uint32_t slot_s, uint32_t byte_pos, uint32_t lut_s, Tree tree,
                                                  uint32_t base, Emit emit) {
    static_assert(SHIFT >= 0 && SHIFT <= 6, "record size");
    constexpr uint32_t AMASK = 0xffffffffu << SHIFT;       // drops the bit-offset bits left below the position
    constexpr uint32_t WMASK = (KVC_LUT_SIZE - 1) << 2;
    const uint32_t end = (base + KVC_VEC_LEN) << 6;
    const uint32_t before = slot_s + byte_pos - 1;         // off = 8, 16, 24 or 32: hi is the word that holds this byte
    uint32_t ptr = before & ~3u;
    uint32_t state = (base << 6) | (26u - ((before & 3u) << 3));
    uint32_t hi = kvc_bswap(kvc_lds32(ptr)), lo = kvc_bswap(kvc_lds32(ptr + 4)), nx = kvc_lds32(ptr + 8);
    ptr += 12;
    auto refill = [&](uint32_t s) {                        // s: the state after a round, 32 more than the bits say
        if (!(s & 32u)) { hi = lo; lo = kvc_bswap(nx); nx = kvc_lds32(ptr); ptr += 4; }
        state = s & ~32u;
    };
    if (!ESC) {
        auto round = [&]() {
            const uint32_t t = __funnelshift_r(lo, hi, state);
            const uint32_t e0 = kvc_lds32(lut_s + ((t >> 16) & WMASK));
            const uint32_t e1 = kvc_lds32(lut_s + (__funnelshift_r(t, 0u, e0) & WMASK));
            const uint32_t s1 = (uint32_t)kvc_dp4a_uu(e0, 1u, (int)state);   // state + byte 0 of e0, off the integer ALU pipe
            emit(e0, (state >> (6 - SHIFT)) & AMASK, state, s1);
            const uint32_t s2 = (uint32_t)kvc_dp4a_uu(e1, 1u, (int)s1);
            emit(e1, (s1 >> (6 - SHIFT)) & AMASK, s1, s2);
            refill(s2);
        };
        // A round emits six symbols at most: the first 21 need no test of the end.  (Attention, 16 x 32768 tokens, 8 x 4 heads: every
        // round tested 670 us, the 21 in threes 656, in sevens 652, all of them 671; one head, 8 x 4096 tokens,
        // without the last: 140, 138, 135.)
#pragma unroll 7
        for (int i = 0; i < (KVC_VEC_LEN - 1) / 6; i++) round();
        do round(); while (state < end);
        return true;
    }
    // The same with a test of each entry; a long code ends its round.  (One lookup per round: one head, rel 0.01 / 0.02,
    // 8 x 4096 tokens, 309 us against 286.)
    bool ok = true;
    // a code longer than the window: on from the node the entry names, one bit at a time
    auto long_code = [&](uint32_t e) {
        uint32_t node = e >> 8, sym = 0;
        bool found = false;
        refill(state + 32u - KVC_LUT_BITS);
        for (int guard = 0; guard < 40; guard++) {
            if (node >= 512u) break;
            const uint32_t nd = tree(node);
            if ((nd & 0xffffu) == KVC_TREE_LEAF) { sym = nd >> 16; found = true; break; }
            const uint32_t bit = (__funnelshift_r(lo, hi, state) >> 29) & 1u;
            refill(state + 31u);
            node = (nd >> (16 * bit)) & 0xffffu;
        }
        ok = ok && found;
        emit((sym << 8) | (1u << 6), (state >> (6 - SHIFT)) & AMASK, state, state + (1u << 6));     // advance byte: one symbol
        state += 1u << 6;
    };
    do {
        const uint32_t t = __funnelshift_r(lo, hi, state);
        const uint32_t e0 = kvc_lds32(lut_s + ((t >> 16) & WMASK));
        if ((e0 & 0xc0u) == 0) { long_code(e0); continue; }
        const uint32_t e1 = kvc_lds32(lut_s + (__funnelshift_r(t, 0u, e0) & WMASK));
        const uint32_t s1 = (uint32_t)kvc_dp4a_uu(e0, 1u, (int)state);
        emit(e0, (state >> (6 - SHIFT)) & AMASK, state, s1);
        if ((e1 & 0xc0u) == 0) { refill(s1 + 16u); if (state < end) long_code(e1); continue; }
        const uint32_t s2 = (uint32_t)kvc_dp4a_uu(e1, 1u, (int)s1);
        emit(e1, (s1 >> (6 - SHIFT)) & AMASK, s1, s2);
        refill(s2);
    } while (state < end);
    return ok;
}

// A consumer for kvc_decode_vector (SHIFT = 0, base = the shared address of the thread's row): the symbols collect in a
// word that is stored when its last byte is known.  One predicated store per word; three byte stores per lookup cost as
// many instructions and, with 32 lanes at 32 places of their rows, three times the bank conflicts.  (The two shifts
// as one wide multiplication: 2.5 % slower in the attention kernel.)  Symbols past position 127 reach at most KVC_DECODE_OVERRUN bytes beyond the row's 128.
struct KvcRowWriter {
    uint32_t cur = 0;
    __device__ __forceinline__ void operator()(uint32_t e, uint32_t a, uint32_t s0, uint32_t s1) {
        const uint32_t syms = e >> 8, sh = a << 3;             // the funnel shifts take the low five bits of the amount
        // (a sum, not an OR: the multiplier pipe can take it from the integer ALU, which takes a warp instruction every other
        // cycle: the grouped attention 970 -> 960 us)
        const uint32_t w = cur + __funnelshift_l(0u, syms, sh), over = __funnelshift_l(syms, 0u, sh);
        const uint32_t left = (s0 ^ s1) & (4u << 6);           // not 0: the position left its word
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p st.shared.u32 [%1], %2;\n\t}"
                     :: "r"(left), "r"(a & ~3u), "r"(w) : "memory");
        cur = left ? over : w;
    }
};

// ---- all lanes of a warp at the same position -----------------------------------------------------------
// The loop above takes what a window holds, one to three symbols, and every lane is at a position of its own.  A consumer that
// multiplies whole words of symbols on the tensor cores wants the opposite: every lane four symbols at a time.  With a fixed number of symbols per lookup
// no position is kept and no end tested; words are put together by byte permutations and go to places known when the kernel is compiled.
//   PAIRS    two symbols per lookup, four per round.  Where few windows hold one code only (two codes at the ends of a bell curve), a lane that meets
//            one falls a symbol behind, up to four: words leave a round late, shifted by what the lane is behind, and every 32 symbols
//            the lanes catch up if one is three or more behind.  Where a lane fell further behind, the warp takes the 32 symbols again, waiting
//            for the last lane at every word.  (A branch for it in every round, taken in every tenth by some lane, cost a third of the attention kernel's time.)
//   SINGLES  one symbol per lookup, for books with longer codes.
// ESC (of PAIRS and SINGLES): some windows hold no complete code.
//   WHOLE    the loop above
enum { KVC_PAIRS = 0, KVC_SINGLES = 1, KVC_WHOLE = 2 };
// Windows with one code or none, of 4096, up to which a book is decoded by pairs: beyond it catching up costs more than the lookups saved.
// (Attention, 16 x 16384 tokens, 8 x 4 heads, pairs and singles: V at rel 0.05 (46 windows) 301 and 341 us, at 0.04 (68) 349 and 341; K, whose lanes have other
// tokens in every step, bears some more: at 0.032 (64) 309 and 348, at 0.028 (96) 318 and 347, at 0.026 (130) 354 and 348; with longer codes than the window, whose
// singles are tested one by one, K per block at 0.02 (82 windows, 51 symbols) 362 and 390.)  Where codes go beyond the window, larger alphabets have more of them
// in the same few channels, and every lane of a warp walks the tree there and falls behind: K per block at 0.018 (82, 57) 381 and 388, at 0.016 (82, 63) 408 and
// 392, at 0.014 (82, 73) 446 and 400, there with 8 heads per KV head 522 and 476; whole rows took 392, 406, 435 and 477.
constexpr uint32_t KVC_PAIRS_LONE = 60, KVC_PAIRS_LONE_ESC = 100;
constexpr int KVC_PAIRS_SYMBOLS_ESC = 60;

struct KvcWay { int way; bool esc; };
__device__ __forceinline__ KvcWay kvc_book_way(const void *book, bool whole) {
    const kvc_book_header *h = reinterpret_cast<const kvc_book_header *>(book);
    if (whole) return {KVC_WHOLE, h->escape != 0};
    const uint32_t lone = h->lone_windows & 0xffffu;
    const bool pairs = (h->lone_windows & 0xffff0000u) != KVC_LONE_KNOWN ? h->escape == 0 && 2 * h->max_len <= KVC_LUT_BITS
                       : h->escape == 0 ? lone <= KVC_PAIRS_LONE : lone <= KVC_PAIRS_LONE_ESC && h->n_symbols <= KVC_PAIRS_SYMBOLS_ESC;
    return {pairs ? KVC_PAIRS : KVC_SINGLES, h->escape != 0};
}
// An entry of these ways' tables: byte 0: 16 - bits of its codes, byte 1: 8 where a pair lacks its second symbol, bytes 2 and 3: the symbols.  No complete
// code: 0 bits, bit 7 of byte 0, and the tree node in bytes 2 and 3.  e: the book's entry; len: bits per symbol.
__device__ __forceinline__ uint32_t kvc_way_entry(uint32_t e, bool pairs, const uint8_t *len) {
    const uint32_t n = (e >> 6) & 3u, bits = e & 63u;
    if (n == 0) return 0x90u | (e << 8 & 0xffff0000u);
    if (!pairs) return (16u - (n == 1 ? bits : len[e >> 8 & 0xffu])) | (e << 8 & 0xff0000u);
    return (16u - bits + (n == 3 ? len[e >> 24] : 0u)) | (n == 1 ? 0x800u : 0u) | (e << 8 & 0xffff0000u);
}
// The tables of two books.  All threads of the CTA call; contains a barrier, between the loads (all of them on their way at once) and
// the stores; the one behind the stores is the caller's.  len: the two books' bits per symbol, 512 bytes.  spare1: a table of single symbols of
// the second book, or null.
__device__ __forceinline__ void kvc_load_ways(uint32_t *lut0, uint32_t *lut1, uint32_t *spare1, const void *book0, const void *book1, bool pairs0, bool pairs1, uint8_t *len, int tid, int nthr) {
    auto at = [](const void *book, int off) { return reinterpret_cast<const uint8_t *>(book) + off; };
    const uint4 *src0 = reinterpret_cast<const uint4 *>(at(book0, KVC_BOOK_OFF_LUT)), *src1 = reinterpret_cast<const uint4 *>(at(book1, KVC_BOOK_OFF_LUT));
    constexpr int N = KVC_LUT_SIZE / 4, AHEAD = 2;
    for (int i = tid; i < 512; i += nthr) len[i] = (uint8_t)__ldg(reinterpret_cast<const uint32_t *>(at(i < 256 ? book0 : book1, KVC_BOOK_OFF_ENC)) + 2 * (i & 255) + 1);
    for (int i = tid; i < N; i += AHEAD * nthr) {
        uint4 a[AHEAD], b[AHEAD];
#pragma unroll
        for (int j = 0; j < AHEAD; j++) { const int k = min(i + j * nthr, N - 1); a[j] = __ldg(src0 + k); b[j] = __ldg(src1 + k); }
        if (i == tid) __syncthreads();                     // (every thread has a first turn: nthr <= N)
#pragma unroll
        for (int j = 0; j < AHEAD; j++) {
            const int k = i + j * nthr;
            if (k >= N) break;
            reinterpret_cast<uint4 *>(lut0)[k] = make_uint4(kvc_way_entry(a[j].x, pairs0, len), kvc_way_entry(a[j].y, pairs0, len), kvc_way_entry(a[j].z, pairs0, len), kvc_way_entry(a[j].w, pairs0, len));
            reinterpret_cast<uint4 *>(lut1)[k] = make_uint4(kvc_way_entry(b[j].x, pairs1, len + 256), kvc_way_entry(b[j].y, pairs1, len + 256), kvc_way_entry(b[j].z, pairs1, len + 256), kvc_way_entry(b[j].w, pairs1, len + 256));
            if (spare1) reinterpret_cast<uint4 *>(spare1)[k] = make_uint4(kvc_way_entry(b[j].x, false, len + 256), kvc_way_entry(b[j].y, false, len + 256), kvc_way_entry(b[j].z, false, len + 256), kvc_way_entry(b[j].w, false, len + 256));
        }
    }
}

__device__ __forceinline__ void kvc_load_tree(uint32_t *tree, const void *book, int tid, int nthr) {
    const uint4 *src = reinterpret_cast<const uint4 *>(reinterpret_cast<const uint8_t *>(book) + KVC_BOOK_OFF_TREE);
    for (int i = tid; i < 512 / 4; i += nthr) reinterpret_cast<uint4 *>(tree)[i] = src[i];
}

// A thread's place in its vector.  The stream's next bits as in kvc_decode_vector; f in the low five bits of s, over whatever the sums leave
// above them: a funnel shift takes no more of it, and a refill is due when the 16s (32 in all) of a round did not carry out of them.
// At most 132 codes of at most 12 bits, or walks of at most 52, are read: a corrupt stream's reads end 0.9 KB behind its vector.
struct KvcCursor {
    uint32_t hi, lo, nx, ptr, s;
    uint32_t behind, last;                                 // PAIRS: 8 bits per symbol the lane is behind, and the word of the round before, its symbols on top
    bool ok;
    __device__ __forceinline__ KvcCursor(uint32_t slot_s, uint32_t byte_pos) {
        const uint32_t before = slot_s + byte_pos - 1;
        ptr = before & ~3u;
        s = 26u - ((before & 3u) << 3);
        hi = kvc_bswap(kvc_lds32(ptr)); lo = kvc_bswap(kvc_lds32(ptr + 4)); nx = kvc_lds32(ptr + 8);
        ptr += 12;
        behind = last = 0u;
        ok = true;
    }
    __device__ __forceinline__ void step(uint32_t n) {
        if (!((s ^ n) & 32u)) { hi = lo; lo = kvc_bswap(nx); nx = kvc_lds32(ptr); ptr += 4; }
        s = n;
    }
    __device__ __forceinline__ uint32_t window() const { return __funnelshift_r(lo, hi, s); }
    __device__ __forceinline__ uint32_t look(uint32_t lut_s, uint32_t t) const { return kvc_lds32(lut_s + (t & ((KVC_LUT_SIZE - 1) << 2))); }
    // the symbol at the window, from the tree node its bits lead to, bit by bit; counts: it is one of the vector's
    __device__ __forceinline__ uint32_t walk(uint32_t node, uint32_t tree_s, bool counts) {
        const KvcTreeShared tree{tree_s};
        uint32_t sym = 0;
        bool found = false;
        step(s + 32u - KVC_LUT_BITS);
        for (int guard = 0; guard < 40 && node < 512u; guard++) {
            const uint32_t nd = tree(node);
            if ((nd & 0xffffu) == KVC_TREE_LEAF) { sym = nd >> 16; found = true; break; }
            const uint32_t bit = window() >> 29 & 1u;
            step(s + 31u);
            node = nd >> (16 * bit) & 0xffffu;
        }
        ok = ok && (found || !counts);
        return sym & 0xffu;
    }
    // two lookups and the step over them; of their symbols the vector has the first `room` bits (8 per symbol) at least
    template <bool ESC> __device__ __forceinline__ void two(uint32_t lut_s, uint32_t tree_s, uint32_t one, uint32_t room, uint32_t &a, uint32_t &b) {
        const uint32_t t = window();
        a = look(lut_s, t >> 16);
        b = look(lut_s, __funnelshift_r(t, 0u, a));
        if (ESC && __builtin_expect((a | b) & 0x80u, 0)) {
            // one of them is no code: its symbol by the tree, as an entry of one symbol and no bits
            if (a & 0x80u) { a = 16u | one | walk(a >> 16, tree_s, room > 0u) << 16; b = look(lut_s, window() >> 16); }
            else { step(s + 16u + (a & 31u)); a = (a & ~31u) | 16u; }
            if (b & 0x80u) b = 16u | one | walk(b >> 16, tree_s, room > 16u - (a >> 8 & 8u)) << 16;
        }
        step(s + a + b);
    }
    // PAIRS: the next two, three or four symbols (any bits on top); now: missing, and 8 bits for each of the four that is not there
    template <bool ESC> __device__ __forceinline__ uint32_t few(uint32_t lut_s, uint32_t tree_s, uint32_t room, uint32_t missing, uint32_t &now) {
        uint32_t a, b, sel = 0x7632u;
        two<ESC>(lut_s, tree_s, 0x800u, room, a, b);
        asm("dp2a.lo.u32.u32 %0, %1, %2, %0;" : "+r"(sel) : "r"(0x02260000u), "r"(a));         // + 0x1130 where a lacks a symbol: {a0, b0, b1, anything}
        // (the sums by byte products, as the shared-memory pipe and the integer ALU are the busiest)
        now = (uint32_t)kvc_dp4a_uu(a, 0x100u, kvc_dp4a_uu(b, 0x100u, (int)missing));
        return __byte_perm(a, b, sel);
    }
    // PAIRS: the next round; returns the word of the round before (any word in the first one).  end: it is the vector's last; what the lane is not
    // behind by lies beyond the vector, where there may be no code at all.
    template <bool ESC> __device__ __forceinline__ uint32_t pairs(uint32_t lut_s, uint32_t tree_s, bool end) {
        uint32_t now;
        const uint32_t c = few<ESC>(lut_s, tree_s, end ? behind : ~0u, behind, now);
        const uint32_t out = __funnelshift_rc(last, c, behind);
        last = c << (now - behind);
        behind = now;
        return out;
    }
    // SINGLES: the next word
    template <bool ESC> __device__ __forceinline__ uint32_t singles(uint32_t lut_s, uint32_t tree_s) {
        uint32_t a, b, c, d;
        two<ESC>(lut_s, tree_s, 0u, ~0u, a, b);
        two<ESC>(lut_s, tree_s, 0u, ~0u, c, d);
        return __byte_perm(__byte_perm(a, b, 0x0062), __byte_perm(c, d, 0x0062), 0x5410);
    }
    // PAIRS: the next one or two symbols of a lane, n bits of them
    template <bool ESC> __device__ __forceinline__ uint32_t take(uint32_t lut_s, uint32_t tree_s, uint32_t &n) {
        const uint32_t a = look(lut_s, window() >> 16);
        if (ESC && (a & 0x80u)) { n = 8u; return walk(a >> 16, tree_s, true); }
        n = 16u - (a >> 8 & 8u);
        step(s + 16u + (a & 31u));
        return a >> 16;
    }
    // PAIRS, between two rounds: lanes that are two or more behind fetch what they lack
    template <bool ESC> __device__ __forceinline__ void catch_up(uint32_t lut_s, uint32_t tree_s) {
        while (behind >= 16u) {
            uint32_t n;
            const uint32_t x = take<ESC>(lut_s, tree_s, n);
            last = __funnelshift_r(last, x, n);
            behind -= n;
        }
    }
    // PAIRS, a lane that fell more than a word behind: back to a place 32 symbols ago, and on from there at the lane's own pace.  put(k, word): word k of 8
    template <bool ESC, class Put> __device__ __forceinline__ void again(uint32_t lut_s, uint32_t tree_s, uint32_t s0, uint32_t ptr0, uint32_t last0, uint32_t behind0, bool end, const Put &put) {
        s = s0; ptr = ptr0;
        hi = kvc_bswap(kvc_lds32(ptr - 12)); lo = kvc_bswap(kvc_lds32(ptr - 8)); nx = kvc_lds32(ptr - 4);
        uint32_t have = 32u - behind0, acc = __funnelshift_rc(last0, 0u, behind0), over = 0u;       // bits that no word has yet
#pragma unroll 1
        for (uint32_t k = 0; k < 8; ) {
            if (have < 32u) {
                uint32_t n;
                const uint32_t y = few<ESC>(lut_s, tree_s, end && k == 7u ? 32u - have : ~0u, 0u, n), x = y << n >> n;
                acc |= x << have;
                over = __funnelshift_lc(x, 0u, have);
                have += 32u - n;
            }
            if (have >= 32u) { put(k, acc); acc = over; over = 0u; have -= 32u; k++; }
        }
        behind = 32u - have;                               // (8 to 32: a word takes 56 bits at most)
        last = __funnelshift_lc(0u, acc, behind);
    }
};
