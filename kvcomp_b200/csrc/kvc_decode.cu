// Blocked Huffman decoder to uint8 codes (kernels.cu:602-719 restated for sm_100a).
//
// One CTA per SM around one copy of the decode table; its workers are pairs of warps, a pair takes one block of 64 vectors
// after the other.  Thread = one vector; decoded symbols go to a shared-memory tile and leave as coalesced stores (K: rows,
// V: transposed back), as codes or, for a reader of values, already dequantised: the codes then never reach memory.  The next
// block's bytes are brought by a bulk copy while the tile goes out, and only the pair's own 64 threads wait for each other.
// Values of 8 sequences x 4096 tokens x 32 heads, device time: K 132 and V 131 us with CTAs of 256 threads that staged, decoded and wrote
// four blocks between barriers of their own, three to an SM with a table each (and the decode loop before the present one); now 97 and 106.
#include "kvc_decode.cuh"

namespace {

constexpr int TILE_STRIDE = 140;          // 128 symbols + KVC_DECODE_OVERRUN rounded up to words, + 1 word; 35 words keep column reads off one bank
constexpr int TILE_BYTES = 64 * TILE_STRIDE; // a tile; the tiles are also the padding a corrupt stream's overrun reads land in
constexpr int MAX_PAIRS = 15;             // named barriers 1 .. 15

struct DecodeSmem {                         // followed by a staging slot per pair (sized at launch), then a tile per pair
    alignas(16) uint32_t lut[KVC_LUT_SIZE];   // the tree, for codes beyond the window, stays in global memory
    uint64_t bar[MAX_PAIRS + 1];
    int dead[MAX_PAIRS + 1];
};
static_assert(sizeof(DecodeSmem) % 16 == 0, "slots are 16-byte aligned");

// VALUES: fp16 values [T, cols, 128] instead of the codes.  The units either do not depend on the channel (m.sc == 0), or
// (K) lie side by side over the channels and cover whole blocks of 64 tokens.  BULK: the stream starts on 16 bytes.
template <bool VALUES, bool BULK>
__global__ void __launch_bounds__(64 * MAX_PAIRS, 1) decode_kernel(
    const uint8_t *__restrict__ encoded, long long encoded_bytes, const uint2 *__restrict__ block_info,
    const uint16_t *__restrict__ thread_info, const void *__restrict__ book, long long nblk, long long cols, int is_k,
    uint32_t max_block, uint32_t slot_bytes, int pairs, uint8_t *__restrict__ codes, kvc_qmeta_dev m, long long H,
    __half *__restrict__ values, int *__restrict__ status, int wait_limit, int starve) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    DecodeSmem &sm = *reinterpret_cast<DecodeSmem *>(smem_raw);
    const int pair = threadIdx.x >> 6, v = threadIdx.x & 63;        // v: the thread's vector of the block
    uint8_t *const slot = smem_raw + sizeof(DecodeSmem) + pair * slot_bytes;
    uint8_t *const tile = smem_raw + sizeof(DecodeSmem) + pairs * slot_bytes + pair * TILE_BYTES;
    const long long row = cols * 128, step = (long long)gridDim.x * pairs, whole = encoded_bytes & ~15ll;
    const KvcTreeGlobal tree(book);
    auto sync = [&]() { asm volatile("bar.sync %0, 64;" :: "r"(pair + 1) : "memory"); };    // the pair's threads
    int flags = 0;
    // a block's record, and from it the bytes [lead, lead + nbytes) of the slot (0 bytes: nothing to decode)
    auto info_of = [&](long long blk) { return blk < nblk ? block_info[blk] : make_uint2(0u, 0u); };
    auto block_of = [&](uint2 bi, uint32_t &off, uint32_t &nbytes, uint32_t &lead, bool &ragged) {
        off = nbytes = lead = 0; ragged = false;
        const uint32_t n = bi.y & 0xffffu;
        const long long end = (long long)bi.x + n;
        if (n > max_block || end > encoded_bytes) { flags |= KVC_FLAG_BAD_STREAM; return; }
        off = bi.x; nbytes = n; lead = (uint32_t)(reinterpret_cast<uintptr_t>(encoded + off) & 15);
        ragged = BULK && end > whole;
    };
    // Bulk copies take whole chunks of 16 bytes, and what lies behind the end of the stream is not the caller's to be read: a
    // block that ends in the stream's last, partial chunk (in the encoder's order the last block) gets that chunk's bytes from the
    // pair's threads, zeroes behind the end.  (The whole block by threads, behind the wait: a call of one block 8.4 us instead of 6.7.)
    auto last_byte = [&]() -> uint8_t { return v < 16 && whole + v < encoded_bytes ? encoded[whole + v] : (uint8_t)0; };
    auto put_last = [&](uint32_t off, uint32_t lead, uint8_t byte) { if (v < 16) slot[(uint32_t)(whole - (off - lead)) + v] = byte; };
    auto start_of = [&](long long blk) { return v && blk < nblk ? (uint32_t)(thread_info[blk * 64 + v - 1] >> 3) : 0u; };
    // by the pair's first thread: one arrival per phase, even for 0 bytes (starve, tests of the bounded waits only: bytes are
    // announced that are never copied)
    auto fetch = [&](uint32_t off, uint32_t nbytes, uint32_t lead, bool ragged) {
        const uint32_t bytes = nbytes ? (lead + nbytes + (ragged ? 0u : 15u)) & ~15u : 0u;
        kvc_mbar_expect_tx(&sm.bar[pair], starve ? 16u : bytes);
        if (bytes && !starve) kvc_bulk_g2s(slot, encoded + off - lead, bytes, &sm.bar[pair]);
    };
    const uint8_t byte = BULK ? last_byte() : (uint8_t)0;      // in flight with the first block's record
    if (BULK && v == 0 && pair < pairs) { kvc_mbar_init(&sm.bar[pair], 1); kvc_mbar_fence_init(); sm.dead[pair] = 0; }
    // neighbouring pairs of the grid take neighbouring blocks
    long long blk = (long long)blockIdx.x * pairs + pair;
    uint32_t off = 0, nbytes = 0, lead = 0;
    bool ragged = false;
    if (pair < pairs) {
        block_of(info_of(blk), off, nbytes, lead, ragged);
        if (BULK && v == 0) fetch(off, nbytes, lead, ragged);
    }
    uint32_t start = pair < pairs ? start_of(blk) : 0u;
    kvc_load_lut(sm.lut, book, threadIdx.x, blockDim.x);
    const bool esc = kvc_book_needs_escape(book);           // uniform over the grid
    if (ragged) put_last(off, lead, byte);
    __syncthreads();                                        // the table and the barriers are in; from here on the pairs go their own ways
    if (pair >= pairs) return;
    uint32_t par = 0;
    for (; blk < nblk; blk += step) {
        const uint2 next = info_of(blk + step);
        bool landed = true;
        if (BULK) {
            // a wait that runs out: the thread does not decode; a barrier whose phase its issuer did not see complete is
            // never armed again, and the pair stops
            landed = kvc_mbar_wait(&sm.bar[pair], par, wait_limit);
            par ^= 1u;
            if (!landed) { flags |= KVC_FLAG_WAIT_TIMEOUT; if (v == 0) sm.dead[pair] = 1; }
        } else {
            if (nbytes) kvc_stage_block(slot, encoded, encoded_bytes, off, nbytes, v, 64);
            sync();
        }
        if (nbytes) {
            bool ok = landed && start < nbytes;
            // the symbols collect in a word that is stored when its last byte is known; symbols past position 127
            // (at most KVC_DECODE_OVERRUN) stay within the row's padding words
            KvcRowWriter put;
            const uint32_t slot_s = kvc_smem_addr(slot), lut_s = kvc_smem_addr(sm.lut), row_s = kvc_smem_addr(tile + v * TILE_STRIDE);
            if (ok) ok = esc ? kvc_decode_vector<true, 0>(slot_s, lead + start, lut_s, tree, row_s, put)
                             : kvc_decode_vector<false, 0>(slot_s, lead + start, lut_s, tree, row_s, put);
            if (!ok) flags |= KVC_FLAG_BAD_STREAM;
        }
        const bool out = nbytes != 0;
        if (ragged && blk + step < nblk) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // put_last, then a bulk copy
        sync();                                             // the tile is complete, the slot free
        if (BULK && sm.dead[pair]) break;
        block_of(next, off, nbytes, lead, ragged);
        if (BULK && v == 0) fetch(off, nbytes, lead, ragged);       // lands while the tile goes out
        if (ragged) put_last(off, lead, last_byte());
        start = start_of(blk + step);
        if (out) {
            if (VALUES && is_k) {                            // thread = 8 channels of every fourth row
                const long long j = blk / cols, col = blk % cols, b = col / H, h = col % H;
                const int c8 = v & 15;
                __half *dst = values + (j * 64) * row + col * 128 + c8 * 8;
                const uint32_t *t4 = reinterpret_cast<const uint32_t *>(tile + c8 * 8);
                if (m.sc != 0) {
                    float mi[8];
                    __half2 sc[4];
                    const long long u = kvc_tok_unit(j * 64, m.tok_div) * m.sj + b * m.sb + h * m.sh + c8 * 8;
#pragma unroll
                    for (int k = 0; k < 8; k++) mi[k] = (float)kvc_load_min(m, u + k) - 8388608.0f;
#pragma unroll
                    for (int k = 0; k < 4; k++) sc[k] = __halves2half2(m.scale[u + 2 * k], m.scale[u + 2 * k + 1]);
#pragma unroll 4
                    for (int r = v >> 4; r < 64; r += 4)
                        *reinterpret_cast<uint4 *>(dst + r * row) = kvc_dequant8(t4[r * (TILE_STRIDE / 4)], t4[r * (TILE_STRIDE / 4) + 1], mi, sc);
                } else {
#pragma unroll 4
                    for (int r = v >> 4; r < 64; r += 4) {
                        float mi; __half2 sc;
                        kvc_row_unit(m, j * 64 + r, b, h, mi, sc);
                        *reinterpret_cast<uint4 *>(dst + r * row) = kvc_dequant8(t4[r * (TILE_STRIDE / 4)], t4[r * (TILE_STRIDE / 4) + 1], mi, sc);
                    }
                }
            } else if (VALUES) {                             // 32 groups of 4 tokens x 8 chunks of 8 channels
                const long long g = blk / (cols * 2), half = blk % (cols * 2), col = half >> 1, b = col / H, h = col % H;
                __half *dst = values + (g * 128) * row + half * 64;
#pragma unroll 2
                for (int i = v; i < 32 * 8; i += 64) {
                    const int tg = i >> 3, c8 = i & 7;
                    uint32_t x[8];
#pragma unroll
                    for (int k = 0; k < 8; k++) x[k] = *reinterpret_cast<const uint32_t *>(tile + (c8 * 8 + k) * TILE_STRIDE + tg * 4);
                    kvc_transpose4x4(x[0], x[1], x[2], x[3]);  // now one word per token: its 4 channels
                    kvc_transpose4x4(x[4], x[5], x[6], x[7]);
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        float mi; __half2 sc;
                        kvc_row_unit(m, g * 128 + tg * 4 + k, b, h, mi, sc);
                        *reinterpret_cast<uint4 *>(dst + (tg * 4 + k) * row + c8 * 8) = kvc_dequant8(x[k], x[4 + k], mi, sc);
                    }
                }
            } else if (is_k) {
                const long long j = blk / cols, col = blk % cols;
                uint8_t *dst = codes + (j * 64) * row + col * 128;
                if ((reinterpret_cast<uintptr_t>(codes) & 15) == 0) {
#pragma unroll
                    for (int k = 0; k < 8; k++) {            // 64 rows x 8 chunks of 16 bytes
                        const int i = v + k * 64, r = i >> 3, c = i & 7;
                        const uint32_t *t4 = reinterpret_cast<const uint32_t *>(tile + r * TILE_STRIDE + c * 16);
                        *reinterpret_cast<uint4 *>(dst + r * row + c * 16) = make_uint4(t4[0], t4[1], t4[2], t4[3]);
                    }
                } else {
                    for (int i = v; i < 64 * 32; i += 64) {
                        int r = i >> 5, w = i & 31;
                        *reinterpret_cast<uint32_t *>(dst + r * row + w * 4) =
                            *reinterpret_cast<const uint32_t *>(tile + r * TILE_STRIDE + w * 4);
                    }
                }
            } else {
                const long long g = blk / (cols * 2), half = blk % (cols * 2);
                uint8_t *dst = codes + (g * 128) * row + half * 64;
                for (int i = v; i < 32 * 16; i += 64) {     // 32 groups of 4 tokens x 16 words of 4 channels
                    const int tg = i >> 4, w = i & 15;
                    uint32_t x0 = *reinterpret_cast<const uint32_t *>(tile + (w * 4 + 0) * TILE_STRIDE + tg * 4);
                    uint32_t x1 = *reinterpret_cast<const uint32_t *>(tile + (w * 4 + 1) * TILE_STRIDE + tg * 4);
                    uint32_t x2 = *reinterpret_cast<const uint32_t *>(tile + (w * 4 + 2) * TILE_STRIDE + tg * 4);
                    uint32_t x3 = *reinterpret_cast<const uint32_t *>(tile + (w * 4 + 3) * TILE_STRIDE + tg * 4);
                    kvc_transpose4x4(x0, x1, x2, x3);          // now one word per token: its 4 channels
                    *reinterpret_cast<uint32_t *>(dst + (tg * 4 + 0) * row + w * 4) = x0;
                    *reinterpret_cast<uint32_t *>(dst + (tg * 4 + 1) * row + w * 4) = x1;
                    *reinterpret_cast<uint32_t *>(dst + (tg * 4 + 2) * row + w * 4) = x2;
                    *reinterpret_cast<uint32_t *>(dst + (tg * 4 + 3) * row + w * 4) = x3;
                }
            }
        }
        sync();                                             // the tile is free
    }
    // the last copy asked for is empty; after a wait that ran out, the one still open may be in flight
    if (BULK && v == 0 && !kvc_mbar_wait(&sm.bar[pair], sm.dead[pair] ? par ^ 1u : par, wait_limit)) flags |= KVC_FLAG_WAIT_TIMEOUT;
    if (flags) atomicOr(status, flags);
}

}  // namespace

// Diagnostics for tests of the bounded waits (kvc_decode_debug): process-wide, read at every launch.
static int g_wait_limit = 0, g_starve = 0;
extern "C" void kvc_decode_debug(int wait_limit, int starve) { g_wait_limit = wait_limit; g_starve = starve; }

// Both outputs' launch; codes or values is null.
static int decode_launch(const char *who, const uint8_t *encoded, int64_t encoded_bytes, const void *block_info,
                         const uint16_t *thread_info, const void *book, int64_t T, int64_t cols, int is_k,
                         uint32_t max_block_bytes, uint8_t *codes, const kvc_qmeta_dev &m, int64_t H, void *values,
                         int32_t *status, kvc_stream_t stream) {
    KVC_REQUIRE(encoded && block_info && thread_info && book && (codes || values) && status, "%s: null pointer", who);
    KVC_REQUIRE(cols > 0 && T >= 0 && encoded_bytes >= 0, "%s: bad shape", who);
    KVC_REQUIRE(T % (is_k ? 64 : 128) == 0, "%s: %s needs a multiple of %d tokens, got %lld", who,
                is_k ? "K" : "V", is_k ? 64 : 128, (long long)T);
    KVC_REQUIRE((reinterpret_cast<uintptr_t>(codes) & 3) == 0 && (reinterpret_cast<uintptr_t>(values) & 15) == 0 &&
                (reinterpret_cast<uintptr_t>(block_info) & 7) == 0 && (reinterpret_cast<uintptr_t>(book) & 15) == 0,
                "%s: misaligned pointer", who);
    const long long nblk = is_k ? (T / 64) * cols : (T / 128) * cols * 2;
    if (nblk == 0) return KVC_OK;
    // a slot holds the largest block plus its alignment lead, in 16-byte chunks, plus the decoder's read-ahead
    const uint32_t max_block = max_block_bytes == 0 || max_block_bytes > 8191u ? 8191u : max_block_bytes;
    const uint32_t slot_bytes = ((max_block + 15u + 15u) & ~15u) + 16u;
    // As many pairs as an SM holds; where the blocks then come in a few rounds, the pairs that this many rounds need: each
    // runs the faster for it.
    const int sms = kvc_sm_count();
    int pairs = MAX_PAIRS;
    while (pairs > 1 && sizeof(DecodeSmem) + pairs * (size_t)(slot_bytes + TILE_BYTES) > 227 * 1024) pairs--;
    const long long rounds = (nblk + (long long)pairs * sms - 1) / ((long long)pairs * sms);
    pairs = (int)((nblk + rounds * sms - 1) / (rounds * sms));
    const size_t smem = sizeof(DecodeSmem) + pairs * (size_t)(slot_bytes + TILE_BYTES);
    const int threads = 64 * (pairs < 4 ? 4 : pairs);       // (the threads beyond the pairs load the table)
    const bool bulk = (reinterpret_cast<uintptr_t>(encoded) & 15) == 0;
    auto *kernel = values ? (bulk ? decode_kernel<true, true> : decode_kernel<true, false>) : (bulk ? decode_kernel<false, true> : decode_kernel<false, false>);
    static kvc_launch_slot slots[4];
    int occ = 0;
    if (int rc = kvc_prepare(slots[(values ? 2 : 0) + bulk], reinterpret_cast<const void *>(kernel), threads, smem, &occ)) return rc;
    KVC_REQUIRE(occ >= 1, "%s: %zu bytes of shared memory do not fit an SM", who, smem);
    const long long ctas = (nblk + pairs - 1) / pairs;
    kernel<<<(unsigned)(ctas < sms ? ctas : sms), threads, smem, kvc_cu(stream)>>>(
        encoded, encoded_bytes, reinterpret_cast<const uint2 *>(block_info), thread_info, book, nblk, cols, is_k,
        max_block, slot_bytes, pairs, codes, m, H, reinterpret_cast<__half *>(values), status,
        g_wait_limit > 0 ? g_wait_limit : KVC_WAIT_LIMIT, g_starve);
    KVC_LAUNCH_OK();
    return KVC_OK;
}

extern "C" int kvc_decode_bounded(const uint8_t *encoded, int64_t encoded_bytes, const void *block_info,
                                  const uint16_t *thread_info, const void *book, int64_t T, int64_t cols, int is_k,
                                  uint32_t max_block_bytes, uint8_t *codes, int32_t *status, kvc_stream_t stream) {
    return decode_launch("kvc_decode", encoded, encoded_bytes, block_info, thread_info, book, T, cols, is_k, max_block_bytes, codes,
                         kvc_qmeta_dev(), 1, nullptr, status, stream);
}

extern "C" int kvc_decode_values(const kvc_cache *c, int64_t T, int64_t B, int64_t H, int is_k, void *out, int32_t *status,
                                 kvc_stream_t stream) {
    KVC_REQUIRE(c && c->q.min_int && c->q.scale && out, "kvc_decode_values: null pointer");
    KVC_REQUIRE(B > 0 && H > 0 && c->q.tok_div > 0, "kvc_decode_values: bad shape");
    KVC_REQUIRE(c->q.min_bytes == 1 || c->q.min_bytes == 2, "kvc_decode_values: min_bytes must be 1 or 2");
    KVC_REQUIRE(c->q.sc == 0 || (is_k && c->q.sc == 1 && c->q.tok_div % 64 == 0),
                "kvc_decode_values: units that depend on the channel are for K only, contiguous over the channels, of whole 64-token blocks");
    return decode_launch("kvc_decode_values", c->encoded, c->encoded_bytes, c->block_info, c->thread_info, c->book, T, B * H, is_k,
                         (uint32_t)(c->max_block_bytes > 0 ? c->max_block_bytes : 0), nullptr, kvc_to_dev(c->q), H, out, status, stream);
}

extern "C" int kvc_decode(const uint8_t *encoded, int64_t encoded_bytes, const void *block_info,
                          const uint16_t *thread_info, const void *book, int64_t T, int64_t cols, int is_k,
                          uint8_t *codes, int32_t *status, kvc_stream_t stream) {
    return kvc_decode_bounded(encoded, encoded_bytes, block_info, thread_info, book, T, cols, is_k, 0u, codes, status, stream);
}
