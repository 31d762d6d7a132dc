// 256-bin symbol histogram and the Huffman codebook build, on the device.
//
// The code assignment reproduces src/huffman.cpp:34-96 (== utils/huffman.py:47-81) bit for
// bit: leaves pushed in ascending symbol order into a binary min-heap keyed on frequency
// only, first popped = left = '0', second popped = right = '1', root-to-leaf path codes.
// The heap discipline (which decides every tie) is the one std::priority_queue and CPython's
// heapq share: push = append + sift up while the parent is strictly larger; pop = walk the
// hole from the root to a leaf always taking the right child unless it is strictly larger
// than the left one, drop the former last element there and sift it up.
#include <cuda.h>
#include <stdarg.h>

#include <mutex>

#include "kvc_common.cuh"

static thread_local char g_err[512] = "";

void kvc_set_error(const char *fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
}

extern "C" const char *kvc_last_error(void) { return g_err; }
extern "C" int kvc_version(void) { return KVC_VERSION; }

int kvc_sm_count() {
    static std::atomic<int> known[KVC_MAX_DEVICES];
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 148;
    const bool keep = dev >= 0 && dev < KVC_MAX_DEVICES;
    if (keep && (n = known[dev].load(std::memory_order_relaxed)) > 0) return n;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 148;
    if (keep) known[dev].store(n, std::memory_order_relaxed);
    return n;
}

// Numbers are given to contexts in the order they are first seen; a context's id is never used again in a process.
int kvc_context() {
    typedef CUresult (*get_id_t)(CUcontext, unsigned long long *);
    static const get_id_t get_id = []() -> get_id_t {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &found) == cudaSuccess && found == cudaDriverEntryPointSuccess)
            return reinterpret_cast<get_id_t>(f);
        cudaGetLastError();
        return nullptr;
    }();
    static std::atomic<unsigned long long> seen[KVC_MAX_CONTEXTS];      // id + 1; 0: free
    unsigned long long id;
    if (!get_id || get_id(nullptr, &id) != CUDA_SUCCESS) return -1;     // (a thread without a context yet)
    for (int i = 0; i < KVC_MAX_CONTEXTS; i++) {
        unsigned long long at = seen[i].load(std::memory_order_relaxed);
        if (at == 0 && seen[i].compare_exchange_strong(at, id + 1, std::memory_order_relaxed)) return i;
        if (at == id + 1) return i;
    }
    return -1;
}

int kvc_prepare(kvc_launch_slot &slot, const void *kernel, int threads, size_t smem, int *occ) {
    static std::mutex mutex;
    const int ctx = kvc_context();
    const bool keep = ctx >= 0 && smem < (1u << 20) && threads % 32 == 0;
    const unsigned long long asked = (unsigned long long)threads / 32 << 48 | (unsigned long long)smem << 8;
    constexpr unsigned long long ASKED = 0xff0000ull << 32 | 0xfffff00ull;
    if (keep) {
        const unsigned long long v = slot.known[ctx].load(std::memory_order_acquire);
        if ((v & 0xff) != 0 && (v & ASKED) == asked) { *occ = (int)(v & 0xff); return KVC_OK; }
    }
    std::lock_guard<std::mutex> lock(mutex);              // the limit never shrinks under another thread's launch
    const size_t limit = keep ? (size_t)(slot.known[ctx].load(std::memory_order_relaxed) >> 28 & 0xfffff) : 0;
    if (smem > limit || limit == 0) {
        KVC_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        KVC_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    }
    KVC_CUDA_OK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, kernel, threads, smem));
    if (keep && *occ > 0 && *occ < 256)
        slot.known[ctx].store(asked | (unsigned long long)(smem > limit ? smem : limit) << 28 | (unsigned)*occ, std::memory_order_release);
    return KVC_OK;
}

extern "C" int kvc_buffer_sizes(int64_t tokens, int64_t hidden, int is_k, int64_t out[4]) {
    KVC_REQUIRE(out != nullptr, "kvc_buffer_sizes: out is null");
    // kernels.cu:898-909: K needs tokens % 64 == 0 and hidden % 128 == 0; V tokens % 128, hidden % 64
    if (is_k) {
        KVC_REQUIRE(tokens % KVC_VEC_PER_BLK == 0, "Context length must be divisible by K_VEC_PER_BLK");
        KVC_REQUIRE(hidden % KVC_VEC_LEN == 0, "Hidden dim must be divisible by K_VEC_LEN");
    } else {
        KVC_REQUIRE(tokens % KVC_VEC_LEN == 0, "Context length must be divisible by V_VEC_LEN");
        KVC_REQUIRE(hidden % KVC_VEC_PER_BLK == 0, "Hidden dim must be divisible by V_VEC_PER_BLK");
    }
    int64_t numel = tokens * hidden;
    out[0] = numel / KVC_VEC_LEN / KVC_VEC_PER_BLK * 8;
    out[1] = numel / KVC_VEC_LEN * 2;
    out[2] = 8;
    out[3] = numel;
    return KVC_OK;
}

namespace {

// ---- histogram: per-warp private bins in shared memory, 16 codes per load ----------------------
__global__ void __launch_bounds__(256) histogram_kernel(const uint8_t *__restrict__ codes, long long n,
                                                        unsigned long long *__restrict__ hist) {
    __shared__ unsigned int sh[8][256];
    const int tid = threadIdx.x, warp = tid >> 5;
    for (int i = tid; i < 8 * 256; i += 256) (&sh[0][0])[i] = 0;
    __syncthreads();
    const long long head = ((16 - (reinterpret_cast<uintptr_t>(codes) & 15)) & 15);   // bytes before alignment
    const long long pre = head < n ? head : n;
    const long long nvec = (n - pre) / 16;
    const uint4 *v = reinterpret_cast<const uint4 *>(codes + pre);
    for (long long i = (long long)blockIdx.x * 256 + tid; i < nvec; i += (long long)gridDim.x * 256) {
        uint4 w = v[i];
        const uint8_t *b = reinterpret_cast<const uint8_t *>(&w);
#pragma unroll
        for (int k = 0; k < 16; k++) atomicAdd(&sh[warp][b[k]], 1u);
    }
    if (blockIdx.x == 0) {   // unaligned head and the tail shorter than 16
        for (long long i = tid; i < pre; i += 256) atomicAdd(&sh[warp][codes[i]], 1u);
        for (long long i = pre + nvec * 16 + tid; i < n; i += 256) atomicAdd(&sh[warp][codes[i]], 1u);
    }
    __syncthreads();
    unsigned int s = 0;
#pragma unroll
    for (int w = 0; w < 8; w++) s += sh[w][tid];
    if (s) atomicAdd(&hist[tid], (unsigned long long)s);
}

// ---- heap, exactly as described at the top of the file -----------------------------------------
// A node is one 64-bit word, (frequency << 10) | id, so that a move in the heap is one load and one
// store; comparisons look at the frequency alone, as the reference's do (ties are decided by position).
struct Heap { unsigned long long *w; int n; };
__device__ __forceinline__ unsigned long long heap_word(long long f, short id) { return ((unsigned long long)f << 10) | (unsigned long long)(id & 0x3ff); }
__device__ __forceinline__ unsigned long long heap_freq(unsigned long long w) { return w >> 10; }

__device__ void heap_sift_up(Heap &hp, int hole, unsigned long long word) {
    while (hole > 0) {
        const int parent = (hole - 1) >> 1;
        const unsigned long long pw = hp.w[parent];
        if (!(heap_freq(pw) > heap_freq(word))) break;
        hp.w[hole] = pw;
        hole = parent;
    }
    hp.w[hole] = word;
}
__device__ void heap_push(Heap &hp, long long f, short id) { hp.n++; heap_sift_up(hp, hp.n - 1, heap_word(f, id)); }
__device__ short heap_pop(Heap &hp, long long *f_out) {
    const unsigned long long top = hp.w[0];
    *f_out = (long long)heap_freq(top);
    const short top_id = (short)(top & 0x3ff);
    int len = --hp.n;
    if (len == 0) return top_id;
    const unsigned long long last = hp.w[len];
    int hole = 0, child = 0;
    while (child < (len - 1) / 2) {
        child = 2 * (child + 1);
        unsigned long long c1 = hp.w[child], c0 = hp.w[child - 1];
        if (heap_freq(c1) > heap_freq(c0)) { child--; c1 = c0; }
        hp.w[hole] = c1;
        hole = child;
    }
    if ((len & 1) == 0 && child == (len - 2) / 2) {
        child = 2 * (child + 1);
        hp.w[hole] = hp.w[child - 1];
        hole = child - 1;
    }
    heap_sift_up(hp, hole, last);
    return top_id;
}

// The heap is a serial chain by contract (its layout decides ties), everything around it is spread over the CTA.  Where all counts together fit 32 bits, its
// words are split into frequencies and ids, two children come with one load, and what a pop has just moved is still in registers when the last word is sifted up.
// (A book of 22 and of 12 symbols: 24.8 and 16.5 us with 64-bit words and the decode table bit by bit, now 18.7 and 12.0; with one thread for the trees as well, 76 us.  Each
// operation by a warp -- the choices of all inner nodes by one ballot, a lane per node -- took 390 cycles a pop.)
constexpr int BOOK_THREADS = 1024;

struct Heap32 {
    uint2 *w;                                               // {frequency, id} of element i at i + 1: an element's children lie in one aligned 128-bit word
    int n;
    __device__ __forceinline__ void sift_up(int hole, uint2 x) {
        while (hole > 0) {
            const int parent = (hole - 1) >> 1;
            const uint2 p = w[parent + 1];
            if (!(p.x > x.x)) break;
            w[hole + 1] = p;
            hole = parent;
        }
        w[hole + 1] = x;
    }
    __device__ __forceinline__ void push(uint32_t freq, uint32_t id) { n++; sift_up(n - 1, make_uint2(freq, id)); }
    __device__ __forceinline__ uint2 pop() {
        const uint2 top = w[1];
        const int len = --n;
        if (len == 0) return top;
        const uint2 last = w[len + 1];
        int hole = 0;
        uint2 moved = make_uint2(0u, 0u);                   // what lies in the hole's parent by now
        while (2 * hole + 2 < len) {
            const uint4 c = *reinterpret_cast<const uint4 *>(w + 2 * hole + 2);
            const bool right = !(c.z > c.x);
            moved = right ? make_uint2(c.z, c.w) : make_uint2(c.x, c.y);
            w[hole + 1] = moved;
            hole = 2 * hole + 1 + (right ? 1 : 0);
        }
        if (2 * hole + 2 == len) {
            moved = w[2 * hole + 2];
            w[hole + 1] = moved;
            hole = 2 * hole + 1;
        }
        if (hole > 0 && moved.x > last.x) {
            w[hole + 1] = moved;
            sift_up((hole - 1) >> 1, last);
        } else w[hole + 1] = last;
        return top;
    }
};

struct BookSmem {
    alignas(16) long long hf[512];
    alignas(16) short hid[512];
    uint16_t first[KVC_LUT_SIZE];    // per window: the symbol that it begins with, and above it the bits of its code (0: no complete code)
    short parent[512];           // of a leaf (its symbol) or an inner node of the Huffman tree: node << 1 | bit
    uint8_t listed[256];         // the symbols that have a code, ascending
    uint32_t aligned[256];       // per listed symbol: its code, first bit on top
    short first_new[256], node0[256];   // per listed symbol: the shortest prefix no earlier symbol has, and its node
    uint32_t warp_sum[BOOK_THREADS / 32];
    int total;
    uint32_t enc_code[256], enc_len[256];
    uint32_t tree[512];          // wide tree: lo16 = child0 (or LEAF), hi16 = child1 (or symbol)
    long long count[256];        // the histogram, fetched by all threads at once
    int n_nodes, n_symbols, min_sym, max_sym, max_len, flags, lone;
    int n_listed, by_walk;       // listed symbols; the trees were built serially: they may lack codes
};

// Exclusive prefix sum of x over the CTA's first 256 threads (the others pass 0); *total receives the sum.
// All threads call; contains barriers.
__device__ uint32_t book_scan(BookSmem &s, uint32_t x, int tid, uint32_t *total) {
    const int lane = tid & 31, warp = tid >> 5;
    uint32_t y = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const uint32_t z = __shfl_up_sync(0xffffffffu, y, o); if (lane >= o) y += z; }
    __syncthreads();
    if (lane == 31) s.warp_sum[warp] = y;
    __syncthreads();
    uint32_t before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < 8; w++) { const uint32_t t = s.warp_sum[w]; if (w < warp) before += t; all += t; }
    *total = all;
    return before + y - x;
}

// insert every code into the decode trees in ascending symbol order
// (build_decode_code_book, src/huffman.cpp:229-252); run by one thread
__device__ void build_trees_serial(BookSmem &s) {      // s.tree was cleared to {NONE, NONE} by the whole CTA
    int n = 2;
    for (int sym = 0; sym < 256; sym++) {
        int len = (int)s.enc_len[sym];
        if (!len) continue;
        int idx = -1, last = -1;
        for (int k = len - 1; k >= 0; k--) {
            int bit = (s.enc_code[sym] >> k) & 1;
            if (idx == -1) idx = bit;
            else {
                uint32_t ch = (s.tree[idx] >> (16 * bit)) & 0xffffu;
                idx = ch == KVC_TREE_NONE ? -1 : (int)ch;
            }
            if (idx == -1) {
                if (n >= 512) { s.flags |= KVC_FLAG_CODE_TOO_LONG; break; }
                uint32_t m = 0xffffu << (16 * bit);
                s.tree[last] = (s.tree[last] & ~m) | ((uint32_t)n << (16 * bit));
                idx = n++;
            }
            last = idx;
        }
        if (idx >= 0) s.tree[idx] = KVC_TREE_LEAF | ((uint32_t)sym << 16);
    }
    s.n_nodes = n;
}

// The same tree, a thread per symbol.  The symbols inserted before symbol i share at most a prefix of m bits with it, so
// its insertion appends the nodes of its prefixes of m + 1 .. length bits, in this order (the one-bit prefixes are
// nodes 0 and 1); a prefix sum over the symbols gives their numbers, and the node of the m-bit prefix is one of the
// first symbol that has this prefix.  Codes beyond 32 bits and trees that do not fit take the serial form.
// All threads call; s.enc_code / enc_len / tree / flags / max_len are set.
__device__ void build_trees(BookSmem &s, int tid) {
    const uint32_t has = tid < 256 && s.enc_len[tid & 255] ? 1u : 0u;
    uint32_t n, total;
    const uint32_t slot = book_scan(s, has, tid, &n);
    if (has) {
        s.listed[slot] = (uint8_t)tid;
        s.aligned[slot] = s.enc_len[tid] <= 32 ? s.enc_code[tid] << (32 - s.enc_len[tid]) : 0u;
    }
    __syncthreads();
    const bool mine = tid < (int)n;
    const uint32_t sym = mine ? s.listed[tid] : 0u, a = mine ? s.aligned[tid] : 0u;
    const int len = mine ? (int)s.enc_len[sym] : 0;
    int m = 1, owner = -1;                              // at least the one-bit prefix is there
    if (mine && len <= 32) {
        for (int j = 0; j < tid; j++) {
            const int c = __clz((int)(a ^ s.aligned[j]));
            if (c > m) { m = c; owner = j; }            // the first one that shares m bits owns the prefix
        }
        m = min(m, len);
    }
    const int fresh = mine ? len - m : 0;
    const uint32_t base = 2u + book_scan(s, (uint32_t)fresh, tid, &total);
    if (tid == 0) { s.n_listed = (int)n; s.by_walk = s.max_len > 32 || total + 2u > 512u; }
    if (s.max_len > 32 || total + 2u > 512u) {
        if (tid == 0) build_trees_serial(s);
        __syncthreads();
        return;
    }
    if (mine) { s.first_new[tid] = (short)(m + 1); s.node0[tid] = (short)base; }
    __syncthreads();
    if (mine) {
        unsigned short *half = reinterpret_cast<unsigned short *>(s.tree);         // child 0 below child 1
        int at = owner < 0 ? (int)(a >> 31) : s.node0[owner] + (m - s.first_new[owner]);
        for (int k = m; k < len; k++) {
            const int next = (int)base + (k - m);
            half[2 * at + ((a >> (31 - k)) & 1u)] = (unsigned short)next;
            at = next;
        }
        s.tree[at] = KVC_TREE_LEAF | (sym << 16);
    }
    if (tid == 0) s.n_nodes = (int)total + 2;
    __syncthreads();
}

// Decode table entry for a KVC_LUT_BITS-bit window w (first stream bit = MSB), 32 bits:
//   byte 0      how far the decoder state advances: (symbols << 6) | bits consumed   (0 = escape)
//   bytes 1..3  up to three complete symbols found in the window, unused bytes 0
// The decoder state is (position in the vector << 6) | bit offset, so one add applies an entry.
// When no code completes inside the window (a code longer than the window, or no code at all)
// byte 0 is 0 and the upper bytes hold the wide-tree node the window's bits lead to; the slow path
// continues from there one bit at a time.
__device__ uint32_t lut_entry(const uint32_t *tree, uint32_t w) {
    uint32_t syms = 0, nsym = 0, used = 0, node = 0;
    int idx = -1, pos = 0;
    while (pos < KVC_LUT_BITS) {
        int bit = (w >> (KVC_LUT_BITS - 1 - pos)) & 1;
        uint32_t ch = idx == -1 ? (uint32_t)bit : ((node >> (16 * bit)) & 0xffffu);
        pos++;
        if (ch == KVC_TREE_NONE || ch >= 512) { idx = -2; break; }     // no such code
        idx = (int)ch;
        node = tree[idx];
        if ((node & 0xffffu) == KVC_TREE_LEAF) {
            syms |= (node >> 16) << (8 * nsym);
            nsym++; used = pos; idx = -1;
            if (nsym == 3) break;
        }
    }
    if (nsym) return (syms << 8) | (nsym << 6) | used;
    return (idx < 0 ? (uint32_t)KVC_TREE_NONE : (uint32_t)idx) << 8;
}

__device__ void write_book(BookSmem &s, uint8_t *book, int tid, int nthr) {
    uint32_t *enc = reinterpret_cast<uint32_t *>(book + KVC_BOOK_OFF_ENC);
    for (int i = tid; i < 256; i += nthr) { enc[2 * i] = s.enc_code[i]; enc[2 * i + 1] = s.enc_len[i]; }
    // reference-format tree: {u8 is_leaf, i8 a, i8 b}; indices and symbols narrowed to 8 bits as
    // include/huffman.h:18-22 does, unset child = -1
    uint8_t *rt = book + KVC_BOOK_OFF_REFTREE;
    for (int i = tid; i < 512; i += nthr) {
        uint32_t nd = s.tree[i];
        uint8_t leaf = 0, a = 0, b = 0;
        if (i < s.n_nodes) {
            if ((nd & 0xffffu) == KVC_TREE_LEAF) { leaf = 1; a = b = (uint8_t)(nd >> 16); }
            else {
                uint32_t c0 = nd & 0xffffu, c1 = nd >> 16;
                a = c0 == KVC_TREE_NONE ? 0xff : (uint8_t)c0;
                b = c1 == KVC_TREE_NONE ? 0xff : (uint8_t)c1;
            }
        }
        rt[3 * i] = leaf; rt[3 * i + 1] = a; rt[3 * i + 2] = b;
    }
    uint32_t *wt = reinterpret_cast<uint32_t *>(book + KVC_BOOK_OFF_TREE);
    for (int i = tid; i < 512; i += nthr) wt[i] = s.tree[i];
    uint32_t *lut = reinterpret_cast<uint32_t *>(book + KVC_BOOK_OFF_LUT);
    // The windows' first symbols, a warp per symbol: a code of up to KVC_LUT_BITS bits has a run of windows.  The others follow from the windows
    // behind; only a window without a complete code walks the tree.
    for (int i = tid; i < KVC_LUT_SIZE / 2; i += nthr) reinterpret_cast<uint32_t *>(s.first)[i] = 0u;
    __syncthreads();
    if (!s.by_walk) for (int i = tid >> 5; i < s.n_listed; i += nthr / 32) {
        const uint32_t sym = s.listed[i], len = s.enc_len[sym];
        if (len > KVC_LUT_BITS) continue;
        const uint32_t at = s.aligned[i] >> (32 - KVC_LUT_BITS);
        for (uint32_t k = tid & 31; k < 1u << (KVC_LUT_BITS - len); k += 32) s.first[at + k] = (uint16_t)(sym | len << 8);
    }
    __syncthreads();
    int no_code = 0, lone = 0;                              // entries whose window holds no complete code, fewer than two of them
    if (tid == 0) s.lone = 0;
    for (int w = tid; w < KVC_LUT_SIZE; w += nthr) {
        uint32_t e = 0, used = 0, nsym = 0;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const uint32_t f = s.first[((uint32_t)w << used) & (KVC_LUT_SIZE - 1)], len = f >> 8;
            if (nsym < (uint32_t)k || len == 0 || used + len > KVC_LUT_BITS) continue;
            e |= (f & 0xffu) << (8 * (k + 1));
            used += len; nsym++;
        }
        e = nsym ? e | nsym << 6 | used : lut_entry(s.tree, (uint32_t)w);
        lut[w] = e;
        no_code |= (e & 0xffu) == 0;
        lone += (e & 0x80u) == 0;
    }
    no_code = __syncthreads_or(no_code);
    if (lone) atomicAdd(&s.lone, lone);
    __syncthreads();
    if (tid == 0) {
        kvc_book_header *h = reinterpret_cast<kvc_book_header *>(book);
        h->n_symbols = s.n_symbols; h->min_sym = s.min_sym; h->max_sym = s.max_sym; h->max_len = s.max_len;
        h->n_nodes = s.n_nodes; h->flags = s.flags; h->lut_bits = KVC_LUT_BITS; h->escape = no_code ? 1 : 0;
        h->lone_windows = KVC_LONE_KNOWN | (uint32_t)s.lone;
    }
}

__global__ void __launch_bounds__(BOOK_THREADS) build_codebook_kernel(const unsigned long long *__restrict__ hist,
                                                                      uint8_t *__restrict__ book) {
    __shared__ BookSmem s;
    const int tid = threadIdx.x;
    const long long count = tid < 256 ? (long long)hist[tid] : 0;
    if (tid < 256) { s.enc_code[tid] = 0; s.enc_len[tid] = 0; }
    if (tid < 512) s.tree[tid] = KVC_TREE_NONE | (KVC_TREE_NONE << 16);
    if (tid == 0) { s.flags = 0; s.max_len = 0; }
    uint32_t nsym;
    const uint32_t slot = book_scan(s, count > 0 ? 1u : 0u, tid, &nsym);
    if (count > 0) { s.listed[slot] = (uint8_t)tid; s.count[slot] = count; }
    const int large = __syncthreads_or(count > 0 && (unsigned long long)count > 0xffffffffu / nsym);      // the sum may not fit 32 bits
    if (tid == 0) {
        s.n_symbols = (int)nsym; s.min_sym = nsym ? s.listed[0] : 0; s.max_sym = nsym ? s.listed[nsym - 1] : 0;
        if (nsym == 0) s.flags |= KVC_FLAG_NO_SYMBOLS;
        short next = 256;
        if (!large) {
            Heap32 hp;
            hp.w = reinterpret_cast<uint2 *>(s.hf); hp.n = 0;
            for (uint32_t i = 0; i < nsym; i++) hp.push((uint32_t)s.count[i], s.listed[i]);
            while (hp.n > 1) {
                const uint2 a = hp.pop(), b = hp.pop();
                s.parent[a.y] = (short)(next << 1); s.parent[b.y] = (short)(next << 1 | 1);
                hp.push(a.x + b.x, (uint32_t)next);
                next++;
            }
        } else {
            Heap hp;
            hp.w = reinterpret_cast<unsigned long long *>(s.hf); hp.n = 0;
            for (uint32_t i = 0; i < nsym; i++) heap_push(hp, s.count[i], (short)s.listed[i]);
            while (hp.n > 1) {
                long long fa, fb;
                const short a = heap_pop(hp, &fa), b = heap_pop(hp, &fb);
                s.parent[a] = (short)(next << 1); s.parent[b] = (short)(next << 1 | 1);
                heap_push(hp, fa + fb, next);
                next++;
            }
        }
        s.total = next - 1;                                 // the root
    }
    __syncthreads();
    if (count > 0) {                                        // a symbol's code, from its leaf up: last bit first
        uint32_t code = 0;
        int len = 0;
        if (nsym == 1) len = 1;                             // utils/huffman.py:42-44: the lone symbol gets '0'
        else for (int nd = tid; nd != s.total; len++) {
            const int up = s.parent[nd];
            if (len < 32) code |= (uint32_t)(up & 1) << len;
            nd = up >> 1;
        }
        s.enc_code[tid] = code; s.enc_len[tid] = (uint32_t)len;
        atomicMax(&s.max_len, len);
        if (len > 32) atomicOr(&s.flags, KVC_FLAG_CODE_TOO_LONG);
    }
    __syncthreads();
    build_trees(s, tid);
    write_book(s, book, tid, BOOK_THREADS);
}

// A reference-format decode tensor (3-byte nodes; child bytes read as unsigned, 0xff = unset)
// -> the same book.  Codes are recovered by walking the tree from both root children.
__global__ void __launch_bounds__(BOOK_THREADS) book_from_tree_kernel(const uint8_t *__restrict__ tree, int n_nodes,
                                                                      uint8_t *__restrict__ book) {
    __shared__ BookSmem s;
    __shared__ uint8_t rt[3 * 256];                         // child bytes reach no further node
    const int tid = threadIdx.x;
    if (tid < 256) { s.enc_code[tid] = 0; s.enc_len[tid] = 0; }
    if (tid < 512) s.tree[tid] = KVC_TREE_NONE | (KVC_TREE_NONE << 16);
    if (tid < 3 * min(n_nodes, 256)) rt[tid] = tree[tid];
    // A thread per node.  Where every node has one parent at most, the first two none, and no symbol two leaves, the leaves find their codes on the way up; any
    // other tensor is walked from the top by one thread, the last leaf of a symbol counting.  (A tree of 43 nodes: 15.0 us with one thread and the table bit by bit, now 8.0.)
    const bool live = tid < n_nodes && tid < 256;
    int *const parents = reinterpret_cast<int *>(s.hf), *const leaves = parents + 256;      // by node and by symbol: how many
    if (tid < 512) parents[tid] = 0;
    if (tid < 256) s.parent[tid] = -1;
    if (tid == 0) { s.flags = 0; s.max_len = 0; s.n_symbols = 0; s.min_sym = 256; s.max_sym = -1; }
    __syncthreads();
    const int c0 = live ? rt[3 * tid + 1] : 0xff, c1 = live ? rt[3 * tid + 2] : 0xff;
    const bool leaf = live && rt[3 * tid] != 0;
    if (live && !leaf) {
        if (c0 != 0xff && c0 < n_nodes) { atomicAdd(&parents[c0], 1); s.parent[c0] = (short)(tid << 1); }
        if (c1 != 0xff && c1 < n_nodes) { atomicAdd(&parents[c1], 1); s.parent[c1] = (short)(tid << 1 | 1); }
    }
    __syncthreads();
    int odd = live && parents[tid] > (tid < 2 ? 0 : 1);
    uint32_t code = 0;
    int len = 0;
    if (leaf) {
        int nd = tid;
        for (; nd >= 2 && len < 256; len++) {
            const int up = s.parent[nd];
            if (up < 0) break;
            if (len < 32) code |= (uint32_t)(up & 1) << len;
            nd = up >> 1;
        }
        if (nd < 2) {                                       // (else: a leaf that no root leads to)
            if (len < 32) code |= (uint32_t)nd << len;
            len++;
            odd |= atomicAdd(&leaves[c0], 1) > 0;
        } else len = 0;
    }
    odd = __syncthreads_or(odd);
    if (!odd && len) {
        s.enc_code[c0] = code; s.enc_len[c0] = (uint32_t)len;
        atomicAdd(&s.n_symbols, 1); atomicMax(&s.max_len, len); atomicMin(&s.min_sym, c0); atomicMax(&s.max_sym, c0);
        if (len > 32) atomicOr(&s.flags, KVC_FLAG_CODE_TOO_LONG);
    }
    __syncthreads();
    if (!odd && tid == 0 && s.n_symbols == 0) { s.min_sym = s.max_sym = 0; s.flags |= KVC_FLAG_NO_SYMBOLS; }
    if (odd && tid == 0) {
        int nsym = 0, mn = 256, mx = -1;
        short *st_node = s.hid; long long *st_code = s.hf;
        int sp = 0;
        if (n_nodes >= 2) { st_node[sp] = 1; st_code[sp] = 1 | (1ll << 40); sp++; st_node[sp] = 0; st_code[sp] = 0 | (1ll << 40); sp++; }
        int guard = 0;
        while (sp && guard++ < 2048) {
            sp--;
            int nd = st_node[sp];
            unsigned long long cl = (unsigned long long)st_code[sp];
            unsigned long long code = cl & 0xffffffffffull, len = cl >> 40;
            if (nd >= n_nodes) continue;
            if (rt[3 * nd]) {
                int sym = rt[3 * nd + 1];
                if (len > 32) s.flags |= KVC_FLAG_CODE_TOO_LONG;
                nsym += s.enc_len[sym] == 0;                // (a symbol at two leaves is one symbol)
                s.enc_code[sym] = (uint32_t)code; s.enc_len[sym] = (uint32_t)len;
                if ((int)len > s.max_len) s.max_len = (int)len;
                if (sym < mn) mn = sym; if (sym > mx) mx = sym;
            } else {
                int c0 = rt[3 * nd + 1], c1 = rt[3 * nd + 2];
                if (c1 != 0xff && sp < 510) { st_node[sp] = (short)c1; st_code[sp] = (long long)((((code << 1) | 1) & 0xffffffffffull) | ((len + 1) << 40)); sp++; }
                if (c0 != 0xff && sp < 510) { st_node[sp] = (short)c0; st_code[sp] = (long long)(((code << 1) & 0xffffffffffull) | ((len + 1) << 40)); sp++; }
            }
        }
        s.n_symbols = nsym; s.min_sym = nsym ? mn : 0; s.max_sym = nsym ? mx : 0;
        if (nsym == 0) s.flags |= KVC_FLAG_NO_SYMBOLS;
    }
    __syncthreads();
    build_trees(s, tid);
    write_book(s, book, tid, BOOK_THREADS);
}

}  // namespace

extern "C" int kvc_histogram(const uint8_t *codes, int64_t n, unsigned long long *hist, kvc_stream_t stream) {
    KVC_REQUIRE(hist != nullptr && (codes != nullptr || n == 0), "kvc_histogram: null pointer");
    KVC_REQUIRE(n >= 0, "kvc_histogram: negative length");
    if (n == 0) return KVC_OK;
    long long want = (n / 16 + 255) / 256;
    long long cap = (long long)kvc_sm_count() * 8;
    unsigned grid = (unsigned)(want < 1 ? 1 : (want > cap ? cap : want));
    histogram_kernel<<<grid, 256, 0, kvc_cu(stream)>>>(codes, n, hist);
    KVC_LAUNCH_OK();
    return KVC_OK;
}

extern "C" int kvc_build_codebook(const unsigned long long *hist, void *book, kvc_stream_t stream) {
    KVC_REQUIRE(hist && book, "kvc_build_codebook: null pointer");
    KVC_REQUIRE((reinterpret_cast<uintptr_t>(book) & 15) == 0, "kvc_build_codebook: book must be 16-byte aligned");
    build_codebook_kernel<<<1, BOOK_THREADS, 0, kvc_cu(stream)>>>(hist, reinterpret_cast<uint8_t *>(book));
    KVC_LAUNCH_OK();
    return KVC_OK;
}

extern "C" int kvc_book_from_tree(const uint8_t *ref_tree, int64_t tree_bytes, void *book, kvc_stream_t stream) {
    KVC_REQUIRE(ref_tree && book, "kvc_book_from_tree: null pointer");
    KVC_REQUIRE(tree_bytes % 3 == 0 && tree_bytes >= 6, "kvc_book_from_tree: a decode tensor holds 3-byte nodes, at least two");
    KVC_REQUIRE(tree_bytes / 3 <= 255, "kvc_book_from_tree: %lld nodes; 8-bit child indices address at most 255", (long long)(tree_bytes / 3));
    KVC_REQUIRE((reinterpret_cast<uintptr_t>(book) & 15) == 0, "kvc_book_from_tree: book must be 16-byte aligned");
    book_from_tree_kernel<<<1, BOOK_THREADS, 0, kvc_cu(stream)>>>(ref_tree, (int)(tree_bytes / 3), reinterpret_cast<uint8_t *>(book));
    KVC_LAUNCH_OK();
    return KVC_OK;
}
