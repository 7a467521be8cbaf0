// Shared host/device infrastructure of libseqtree_b200: error plumbing, the per-device
// context (stream, grow-only device workspace, pinned staging), and the device-resident
// sequence set.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>
#include <functional>
#include <map>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/seqtree_b200.h"

namespace stb {

// ----------------------------------------------------------------------------- errors -------
// Every failure inside the library is a StError carrying the C-ABI code and the exact message
// the reference raises for the same condition; the extern "C" wrappers turn it into st_error.
struct StError : std::runtime_error {
    int32_t code;
    StError(int32_t c, const std::string& m) : std::runtime_error(m), code(c) {}
};

[[noreturn]] inline void fail(int32_t code, const std::string& msg) { throw StError(code, msg); }

#define STB_CUDA(expr)                                                                        \
    do {                                                                                      \
        cudaError_t e_ = (expr);                                                              \
        if (e_ != cudaSuccess)                                                                \
            ::stb::fail(e_ == cudaErrorMemoryAllocation ? ST_ENOMEM : ST_ECUDA,               \
                        std::string("CUDA error: ") + cudaGetErrorString(e_) + " at " +       \
                            __FILE__ + ":" + std::to_string(__LINE__));                      \
    } while (0)

// Launch bookkeeping: the number of kernels the last call launched and the main variant.
void note_launch(const char* kernel_name, int count = 1);
void reset_launches();

// Host-side phase tracing.  Every Phase opens an NVTX range (visible to Nsight tools, free
// otherwise); with SEQTREE_B200_TRACE=1 in the environment the wall time of each phase is also
// recorded and trace_report() prints one line per call to stderr.
struct Phase {
    const char* name;
    double t0;
    explicit Phase(const char* n);
    ~Phase();
};
void trace_report(const char* call);

// ----------------------------------------------------------------------------- context ------
// A device buffer that only grows; reused across calls so steady-state calls allocate nothing.
struct DevBuf {
    void* ptr = nullptr;
    size_t cap = 0;
    void* get(size_t bytes);
    template <class T>
    T* as(size_t count) { return static_cast<T*>(get(count * sizeof(T))); }
    // Grows to at least `bytes`, keeping the first `keep` bytes (device-to-device on `stream`).
    void* grow_keep(size_t bytes, size_t keep, cudaStream_t stream);
    void release();  // frees the memory now (owners that do not live until exit)
    ~DevBuf();
};

struct Context;

// Stream-ordered memory from pools of the library's own: calls on several streams each get theirs, a
// captured call gets its allocation as graph nodes, and a bounded amount stays cached for the next.  Freed
// on the stream it was taken for, unless keep() hands it (taken to_keep) to an owner, which gives it to
// kept_free() once nothing reads it.
void kept_free(void* ptr, size_t bytes);

struct StreamScratch {
    void* ptr = nullptr;
    cudaStream_t stream = nullptr;
    StreamScratch() = default;
    StreamScratch(int device, size_t bytes, cudaStream_t st) { take(device, bytes, st); }
    void take(int device, size_t bytes, cudaStream_t st, bool to_keep = false);
    void* keep() {
        void* p = ptr;
        ptr = nullptr;
        return p;
    }
    ~StreamScratch() {
        if (ptr) cudaFreeAsync(ptr, stream);
    }
    StreamScratch(const StreamScratch&) = delete;
    StreamScratch& operator=(const StreamScratch&) = delete;
};

// The buffers of a set's plans: they grow, and go with their owner (whose destructor frees device memory of its
// own first, which waits for the kernels that still read them).  From the library's pools, as plans come
// and go with their sets: cudaMalloc after such a free had to map memory again, 1 to 2 ms in a first
// call on new sets (B200).
struct OwnedBuf {
    void* ptr = nullptr;
    size_t cap = 0;
    void* get(size_t bytes, cudaStream_t stream);
    template <class T>
    T* as(size_t count, cudaStream_t stream) { return static_cast<T*>(get(count * sizeof(T), stream)); }
    OwnedBuf() = default;
    OwnedBuf(const OwnedBuf&) = delete;
    OwnedBuf& operator=(const OwnedBuf&) = delete;
    ~OwnedBuf() { kept_free(ptr, cap); }
};

struct StreamNow {  // a call's stream, looked at once
    cudaStream_t stream;
    unsigned long long id = 0;
    bool capturing = false;
    explicit StreamNow(cudaStream_t s);
    StreamNow(const Context& ctx, cudaStream_t s);  // (nothing to look at for the context's own stream)

private:
    StreamNow(cudaStream_t s, unsigned long long known) : stream(s), id(known) {}
};

// Something made on one stream (a plan) that calls on any stream then read: other streams wait for it on the
// device, nothing on the host does.  (Transient sets' calls are all on the context's stream.)
struct Made {
    void on(cudaStream_t stream);      // everything enqueued on `stream` so far
    void need(const StreamNow& now);   // what follows on the stream may read it
    void need(cudaStream_t stream) {
        if (event) need(StreamNow(stream));
    }
    Made() = default;
    Made(const Made&) = delete;
    Made& operator=(const Made&) = delete;
    ~Made() {
        if (event) cudaEventDestroy(event);
    }

private:
    cudaEvent_t event = nullptr;
    unsigned long long stream_id = 0;  // the last stream known to be behind it
};

struct Context {
    int device = 0;
    std::mutex mu;              // serialises calls on this device
    cudaStream_t stream = nullptr;
    unsigned long long stream_id = 0;
    int num_sms = 148;
    int max_smem_optin = 0;
    // Small device word area for error reporting, with a pinned host mirror.  Word 0: first
    // invalid symbol of an encode; words 6-7: make_pair's invalid symbols; word 8: a bounded wait gave up; word 9: an int32 overflow;
    // words 16-23: byte-presence bitmaps of two sets.  Words 6-15 are cleared before and read after each
    // host call.
    int64_t* flags_d = nullptr;
    int64_t* flags_h = nullptr;
    // second stream and events of the host calls that overlap the result copy with the kernels
    cudaStream_t copy_stream = nullptr;
    cudaEvent_t block_ev[8] = {};
    // the last use of the scratch and tables below by a call on a caller's stream (ScratchTurn)
    Made scratch;
    // named scratch, grow-only
    DevBuf out_buf, q_codes, r_codes, table_buf, prior_buf, ftab_buf, work_a, work_b, work_c;
    // sparse output: unsorted hit keys and scores, sorted keys, radix-sort scratch
    DevBuf sp_keys, sp_vals, sp_sorted, sp_temp;
    // candidate lists of the learned-proposal kernel; the threshold form's table
    DevBuf topk_cand, prop_thr, prop_items;
    std::vector<uint8_t> prop_thr_key;
    // bf16 operands of the training GEMM, packed in the tensor-core layout
    DevBuf gemm_a, gemm_b;
    // block of make_pair's sets and its pinned upload block (1 MiB, made on first use)
    DevBuf pair_buf;
    uint8_t* stage_h = nullptr;
    // storage of the transient sets made by the host-buffer entry points
    DevBuf tq[3], tr[3];  // bytes, offsets, lengths
    // kept_table's tables by content, and their blocks
    std::map<std::vector<int32_t>, int32_t*> tables;
    DevBuf table_blocks[16];
    // plans reused by transient sets (rebuilt in place for every call)
    std::shared_ptr<void> tmp_query_plan, tmp_ref_plan, tmp_wave_plan[2];
    // ref plan of the tuner's trials on a resident set (each trial is waited for)
    std::shared_ptr<void> trial_ref_plan;
    std::shared_ptr<void> tmp_strip_query_plan, tmp_strip_ref_plan, tmp_dist_plan[2];
    // query plan of a row block (sparse calls whose hits are taken in several blocks)
    std::shared_ptr<void> tmp_block_plan;
    // sparse result of the host-buffer sparse call (an st_hits_s)
    std::shared_ptr<void> tmp_hits;
};

// Context of the current CUDA device (created on first use).  Fails with ST_ENODEV when no
// device is usable.
Context& context();

// A call's turn with the context's scratch and tables: what it enqueues while this lives comes after the
// last such call's kernels, whatever stream they are on.  Nothing orders a graph's replays with later
// calls, so a captured call takes memory of its own instead (`own`, which becomes the graph's).
struct ScratchTurn {
    Context& ctx;
    const StreamNow now;
    ScratchTurn(Context& c, cudaStream_t s);
    ~ScratchTurn();
    ScratchTurn(const ScratchTurn&) = delete;
    ScratchTurn& operator=(const ScratchTurn&) = delete;
    template <class T>
    T* as(DevBuf& shared, size_t count, StreamScratch& own) {
        if (!now.capturing) return shared.as<T>(count);
        own.take(ctx.device, count * sizeof(T), now.stream);
        return static_cast<T*>(own.ptr);
    }
};

// Raises `kernel`'s dynamic shared-memory limit to `bytes` on the current device, once per
// (device, kernel, size).  The attribute belongs to a device, so a process that uses several
// devices needs the call on each of them.
void ensure_smem_limit(const void* kernel, size_t bytes);

// Fails while `stream` is being captured: for what a call makes and keeps, which a capture would only record.
void refuse_capture(cudaStream_t stream);

// Host -> device copy of per-call tables or plans.  Refuses to run while `stream` is being
// captured into a CUDA graph: the captured copy would read host memory that is gone when the
// graph is replayed.  Plans and tables are cached, so a call made once before capturing leaves
// nothing to upload inside the capture.
void h2d(void* dst, const void* src, size_t bytes, cudaStream_t stream);

// A small table (at most 1,024 words) on the device, by content.  The first 1,024 of a device are uploaded once
// and never rewritten, so calls on any streams and captured graphs may read them at any time; a
// further one is uploaded into `spare` for its call alone.
const int32_t* kept_table(Context& ctx, const std::vector<int32_t>& v, cudaStream_t stream, StreamScratch& spare);

inline bool table_kept(const Context& ctx, const std::vector<int32_t>& v) { return ctx.tables.count(v) != 0; }

// Byte-exact content cache: returns true when `bytes` equals what was uploaded last time
// under `slot`, so re-uploads of unchanged tables are skipped.
bool same_as_last(std::vector<uint8_t>& slot, const void* data, size_t bytes);

// ----------------------------------------------------------------------------- tuning -------
// Measured choice among `n` launch variants that produce identical results.  The first time `key`
// is seen on a device (and tuning is on and `stream` is not being captured), every variant runs
// once untimed and then 3-9 times timed with CUDA events on `stream` (more while the runs are
// short), and the one with the fastest median is cached; every
// call ends with the chosen variant's results in place.  Later calls with the key run the cached
// choice directly.  Tuning is off with SEQTREE_B200_TUNE=0; then, and while `stream` is being
// captured before the key was tuned, `run(fallback)` runs (`fallback` may be -1, the caller's
// static choice).
// `best_ms`, when given, gets the choice's time if this call measured it.
int tuned_run(const std::string& key, int n, int fallback, const std::function<void(int)>& run,
              cudaStream_t stream, float* best_ms = nullptr);
// Records a choice for `key` unless it has one.
void tuned_keep(const std::string& key, int choice);
// The cached choice for `key` on the current device, or -1.
int tuned_lookup(const std::string& key);
// False when SEQTREE_B200_TUNE=0 switched measured tuning off.
bool tuning_enabled();
// log2 bucket of a size, for shape keys.
inline int size_bucket(int64_t n) {
    int b = 0;
    while (n > 1) {
        n >>= 1;
        ++b;
    }
    return b;
}

// ----------------------------------------------------------------------------- sets ---------
// A sequence set resident on one device: the concatenated (encoded or raw) bytes, offsets and
// lengths, plus host-side length metadata used to plan launches.
}  // namespace stb

struct st_seqset_s {
    int device = 0;
    int32_t alphabet = -1;      // ST_ALPHABET_* or -1 for raw bytes
    int64_t count = 0;
    int64_t total = 0;          // bytes
    int32_t max_len = 0;
    std::vector<int64_t> h_off; // count + 1
    std::vector<int32_t> h_len; // count
    uint8_t* d_bytes = nullptr; // encoded codes (alphabet >= 0) or raw bytes, +64 B padding
    int64_t* d_off = nullptr;
    int32_t* d_len = nullptr;
    bool owns = true;           // false: storage borrowed from the context (transient set)
    uint64_t uid = 0;           // unique per set; plans record the uid they were built for
    // plan caches (opaque; transient sets share the context's)
    std::shared_ptr<void> gb_query_plan, gb_ref_plan, wave_plan, strip_query_plan, strip_ref_plan;
    std::shared_ptr<void> dist_plan;
    int64_t align_calls = 0;    // alignment calls so far (a set is planned for on its second)
    ~st_seqset_s();
};

// A thresholded sparse result resident on one device: CSR rows over the query set.
struct st_hits_s {
    int device = 0;
    int64_t rows = 0, cols = 0, nnz = 0;
    uint64_t cap_hint = 0;       // hit-buffer size that the next call starts from
    int64_t block_rows_hint = 0; // query rows per block the last call needed (0: one block)
    stb::DevBuf indptr;          // rows + 1 int64
    stb::DevBuf ref_ids;         // nnz int32, ascending within a row
    stb::DevBuf scores;          // nnz int32
    ~st_hits_s() {
        indptr.release();
        ref_ids.release();
        scores.release();
    }
};

namespace stb {

// Uploads and encodes `s` onto the current device.  When `bad_index` is non-null the first
// invalid symbol's byte index is returned there (or -1) instead of failing, so a caller can
// order errors across two sets exactly as the reference does.
// `storage` (three buffers: bytes, offsets, lengths) makes a transient set that borrows
// context memory instead of allocating.
st_seqset_s* make_seqset(const st_strings* s, int32_t alphabet, cudaStream_t stream,
                         int64_t* bad_index, char* bad_char, DevBuf* storage = nullptr);

// Both sets of a host-buffer call as transient sets, in one upload (of up to 1 MiB) and one launch.
// Nothing waits for the symbol check: an invalid symbol is stored as code 0 (so every later kernel
// indexes its tables in range) and bad[t], two device words that hold 0 before, gets the complement
// of set t's first invalid byte index for the caller to read after its final synchronisation.
void make_pair(const st_strings* const in[2], int32_t alphabet, cudaStream_t stream, unsigned long long* bad,
               std::unique_ptr<st_seqset_s> sets[2]);

int32_t alphabet_size(int32_t alphabet);

// The first `rows` sequences of `s` as a set that borrows its device storage (no copy, no
// allocation; plans go to the context's transient slots).  Valid while `s` lives.
std::unique_ptr<st_seqset_s> row_view(const st_seqset_s& s, int64_t rows);

inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

}  // namespace stb
