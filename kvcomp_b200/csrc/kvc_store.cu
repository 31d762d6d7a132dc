// A store in one call: quantise, book, encode, the rows that stay rows, and one copy that brings back what all of them report
// (models/cache/kvcomp_encode.py:60-207 makes these calls one by one, with a wait behind each).
//
// The kernels are those of the single calls.  What is saved is around them: one memset for the report, the histogram and the encoder's states
// instead of three, no arguments converted and no temporary made between two launches, and nothing that waits.
#include <string.h>

#include "kvc_common.cuh"

namespace {

constexpr int64_t REPORT_BYTES = 32, HIST_BYTES = 256 * 8;
int64_t pad16(int64_t n) { return (n + 15) & ~15ll; }

}  // namespace

// scratch: {encoder's bytes, largest block, quantiser's flags, encoder's flags}, histogram, encoder's workspace, quantiser's workspace
extern "C" int64_t kvc_store_scratch(int mode, int batch_shared, int64_t T, int64_t B, int64_t H, int64_t block, int64_t enc_T, int is_k) {
    return REPORT_BYTES + HIST_BYTES + pad16(kvc_encode_workspace(enc_T, B * H, is_k)) + pad16(kvc_quantize_workspace(mode, batch_shared, T, B, block)) + 16;
}

extern "C" int kvc_stream_wait(kvc_stream_t stream) {
    KVC_CUDA_OK(cudaStreamSynchronize(kvc_cu(stream)));
    return KVC_OK;
}

extern "C" int kvc_store_packed(const kvc_store_args *args, kvc_stream_t stream) {
    KVC_REQUIRE(args, "kvc_store_packed: null pointer");
    kvc_store_args a;
    memcpy(&a, args, sizeof(a));                            // (wherever the caller packed them)
    KVC_REQUIRE(a.scratch && (a.book || (a.enc_table && a.T == 0)) && a.report && a.T >= 0 && a.enc_T >= 0, "kvc_store_packed: null pointer or bad shape");
    KVC_REQUIRE((reinterpret_cast<uintptr_t>(a.scratch) & 15) == 0 && a.scratch_bytes >= kvc_store_scratch(a.mode, a.batch_shared, a.T, a.B, a.H, a.block, a.enc_T, a.is_k),
                "kvc_store_packed: scratch must be 16-byte aligned and hold what kvc_store_scratch says");
    KVC_REQUIRE(a.T > 0 || !a.build, "kvc_store_packed: nothing to build a book from");
    KVC_REQUIRE(a.T > 0 || a.enc_T > 0, "kvc_store_packed: nothing to store");     // (kvc_encode has no codes to look at then and refuses the call)
    KVC_REQUIRE(a.kept_rows >= 0 && a.kept_rows <= a.T && a.rest_rows >= 0, "kvc_store_packed: bad row counts");
    KVC_REQUIRE(a.rest_rows == 0 || (a.heads && a.T > 0 && a.rest && a.rest_rows <= a.x_tokens - a.T),
                "kvc_store_packed: %lld rows behind the first %lld of %lld tokens", (long long)a.rest_rows, (long long)a.T, (long long)a.x_tokens);
    kvc_qmeta kept_units = {};
    int64_t n_units = 0;
    if (a.kept_rows > 0) {
        if (int rc = kvc_qmeta_make(a.mode, a.batch_shared, a.T, a.B, a.H, a.D, a.block, &kept_units, &n_units)) return rc;
        KVC_REQUIRE(a.kept && a.kept_rows % kept_units.tok_div == 0, "kvc_store_packed: %lld kept rows are not whole units of %d tokens", (long long)a.kept_rows, kept_units.tok_div);
    }
    KVC_REQUIRE(a.enc_T == 0 || (a.base_offset >= 0 && a.base_offset <= 0xffffffffll),
                "kvc_store_packed: a block's offset has 32 bits, the stream begins at %lld", (long long)a.base_offset);
    uint8_t *const scratch = reinterpret_cast<uint8_t *>(a.scratch);
    unsigned long long *const total = reinterpret_cast<unsigned long long *>(scratch);
    int32_t *const quant_status = reinterpret_cast<int32_t *>(scratch + 16), *const enc_status = reinterpret_cast<int32_t *>(scratch + 24);
    unsigned long long *const hist = a.build ? reinterpret_cast<unsigned long long *>(scratch + REPORT_BYTES) : nullptr;
    uint8_t *const enc_ws = scratch + REPORT_BYTES + HIST_BYTES;
    const int64_t enc_bytes = kvc_encode_workspace(a.enc_T, a.B * a.H, a.is_k);
    uint8_t *const quant_ws = enc_ws + pad16(enc_bytes);
    cudaStream_t s = kvc_cu(stream);
    KVC_CUDA_OK(cudaMemsetAsync(scratch, 0, (size_t)(REPORT_BYTES + HIST_BYTES + enc_bytes), s));
    if (a.T > 0 && a.heads) {
        if (int rc = kvc_quantize_heads(a.x, a.cos_, a.sin_, a.cos_batch_stride, a.B, a.H, a.x_tokens, a.T, a.D, a.mode, a.batch_shared, a.block, a.rel,
                                        a.codes, a.min_int, a.min_bytes, a.scale, hist, quant_status, stream)) return rc;
    } else if (a.T > 0) if (int rc = kvc_quantize(a.x, a.T, a.B, a.H, a.D, a.mode, a.batch_shared, a.block, a.rel, a.codes, a.min_int, a.min_bytes, a.scale, hist,
                                     quant_ws, scratch + a.scratch_bytes - quant_ws, quant_status, stream)) return rc;
    if (a.build) if (int rc = kvc_build_codebook(hist, a.book, stream)) return rc;
    if (a.enc_T > 0)
        if (int rc = kvc_encode_zeroed(a.enc_codes, a.enc_T, a.B * a.H, a.is_k, a.enc_table ? a.enc_table : reinterpret_cast<const uint8_t *>(a.book) + KVC_BOOK_OFF_ENC,
                                       a.enc_table ? a.n_entries : 256, (uint32_t)a.base_offset,
                                       a.block_info, a.thread_info, a.encoded, a.encoded_capacity, total, enc_ws, enc_bytes, enc_status, stream)) return rc;
    KVC_CUDA_OK(cudaMemcpyAsync(a.report, scratch, REPORT_BYTES, cudaMemcpyDeviceToHost, s));
    if (a.rest_rows > 0)                                     // (behind the copy: the report is on its way while they are written)
        if (int rc = kvc_rope_store_rows(a.x, a.cos_, a.sin_, a.rest, a.B, a.H, a.x_tokens, a.T, a.rest_rows, a.D, a.cos_batch_stride, stream)) return rc;
    if (a.kept_rows > 0) {
        kvc_qmeta &q = kept_units;
        const int64_t first = (a.T - a.kept_rows) / q.tok_div * q.sj;       // unit of the first kept token
        q.min_int = reinterpret_cast<uint8_t *>(a.min_int) + first * a.min_bytes;
        q.scale = reinterpret_cast<uint16_t *>(a.scale) + first;
        q.min_bytes = a.min_bytes;
        if (int rc = kvc_dequant(a.codes + (a.T - a.kept_rows) * a.B * a.H * a.D, &q, a.kept_rows, a.B, a.H, a.D, a.kept, stream)) return rc;
    }
    return KVC_OK;
}
