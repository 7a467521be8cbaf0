// Dense single-gap-block penalty matrix on sm_100a.
//
// Reference arithmetic (seqtree src/gapblock.cpp:39-62): for a pair (q, r) with L = min(m,n),
// d = |m-n|, the layout whose block opens at column i of the shorter sequence costs
//     pre[i] + suf[i] + prior[i]     (prefix on diagonal 0, suffix on diagonal d)
// and the score is the minimum over i in [0, L] plus gap_open + (d-1)*gap_extend; at d == 0
// it is the plain substitution sum.  With P0[j] = pen on diagonal 0 and Pd[j] = pen on
// diagonal d, pre[i] + suf[i] = S + C[i] where S = sum_j Pd[j] and C[i] = sum_{j<i}(P0 - Pd),
// so one forward sweep visits every block position -- that is the form computed here.  The
// result is the same integer as the reference's (integer sums, no reassociation hazard while
// the reference itself does not overflow int32).
//
// Fast path (every length <= 64, min(m,n) * max_pen <= 8191, no negative penalty):
//   * The minimum runs along the sweep: A[i] = pre[i] + prior[i] and B[i] = the best layout whose
//     block has opened at or before i, charged up to column i:
//         A += P0[j] + (prior[j+1] - prior[j]);   B = min(B + Pd[j], A)
//     -- one three-input add and one DPX __viaddmin_s16x2 for two queries packed int16x2.
//   * Queries of one length travel in quads: a profile word holds the four queries' penalties
//     against one residue, 8 bits each (one LDS.32 = four pair-cells per lane), split into two
//     int16x2 words by a PRMT (odd bytes) and an IMAD (w - 256 * odd) on the otherwise idle FMA
//     pipe.  Penalties above 255 use two 16-bit words instead (WIDE).  A CTA's four quads form a
//     slice; its profile is [row][quad][32 words], one pass over the banks per quad.
//   * Refs are cut into chunks of RC columns (original order); inside a chunk they are sorted by
//     length and taken 32 at a time, one per lane, whatever their lengths: each lane has its own
//     diagonal, a ref's code rows past its end hold a code whose penalties are 0, and the prior's
//     steps past a layout's last position are 0, so the positions past a lane's own end change
//     nothing.  (Warps of one length only were 82 % full.)  The codes are laid out per warp task
//     as [j][lane] bytes holding 4 * code, a byte offset into a profile row.
//   * A CTA owns (chunk, slice).  Two bulk (TMA) copies stage the slice's profile and the chunk's
//     code slab, completing on one mbarrier.  Every lookup is LDS [lane register + immediate].
//   * Dense results go through a shared tile so that the global stores are coalesced in the
//     original column order; the per-(m,n) term (prior minimum + gap cost) is added there.
//   Measured, B200 at 1965 MHz, against the form with 16-bit pair words, three ALU operations per
//   pair-cell and warps of one length: 9,973 x 50,021 junctions of 8-25, BLOSUM62, dense 2.10 ->
//   0.91 ms; 100,000 x 1,000,000 thresholded at 24 366 -> 139 ms.  The sweep is bound by issue
//   slots (78-82 % issue active; ALU 57-63 %, FMA 53-60 %, shared wavefronts 75 % of a cycle).
// General path: one thread per pair in int32 for any lengths and penalty magnitudes.
//
// Thresholded sparse form (for matrices too large to hold densely): the same kernels keep only
// the cells with score <= max_penalty and turn them into CSR rows (indptr, ref ids, scores):
// exactly the entries of the dense matrix's rows that pass the threshold, in ref order.  The fast
// kernel tests its results in registers, marks hits in a bitmap of the tile and writes them in
// column order; the general kernel appends (query << shift | ref, score) with one atomic per warp
// and the hits are radix-sorted.
#include <algorithm>
#include <cstdlib>
#include <map>
#include <type_traits>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include "common.cuh"
#include "sparse.cuh"

namespace stb {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kRow = 32;        // words of one quad in a profile row
constexpr int kQuads = 4;       // quads per slice
constexpr int kSliceQ = 4 * kQuads;
constexpr int kNullCode = 31;   // a residue past a ref's end: its profile column is 0
constexpr int kMaxSum = 8191;   // largest sum of penalties along a pair that the fast form takes
constexpr int kMaxHalf = 32767; // largest value of a packed half
constexpr int kMaxSpread = 8;   // lengths of one warp task differ by at most this
constexpr int kTileW = 2 * kQuads + 1;  // tile words per column: 8 results and the (m, n) term
static_assert(kWarps == 2 * kQuads, "the dense write-out gives each result word one warp");

// ---------------------------------------------------------------------------- plans ---------
// Plans depend only on the lengths (and codes) of a set, so a device-resident set builds them
// once; transient sets (host-buffer calls) rebuild them in place inside the context's plan
// objects, whose device buffers only grow.  What a resident set keeps -- its plans, a ref plan for each
// chunk width it is called with, a profile for each of the first four penalty grids -- is never written
// again, so calls on any streams and captured graphs may read it as long as the set lives.  Further grids
// share a fifth profile: it changes only when the device is idle, and captured calls are refused it.
struct Profile {
    std::vector<uint8_t> key;            // (A, word width, penalty grid) it was built for
    OwnedBuf buf;                        // [row][quad][32] uint32 (twice the words when WIDE)
    Made made;
};
constexpr size_t kMaxProfiles = 5;  // the last one changes hands

struct QueryPlan {
    uint64_t uid = 0;                    // set the plan was built for
    int64_t r0 = 0, r1 = -1;             // its rows [r0, r1) (r1 = -1: the whole set)
    std::vector<int4> quads;             // original indices (-1 marks an empty slot)
    std::vector<int4> slices;            // (first quad, quads, length, profile row offset)
    int64_t prof_rows = 0;               // profile rows of all slices
    OwnedBuf d_plan;                     // quads, then slices
    Made made;
    std::vector<std::unique_ptr<Profile>> profiles;
};

struct RefPlan {
    uint64_t uid = 0;
    int rc = 0;                          // columns per chunk
    int64_t nchunks = 0;
    int64_t ntasks = 0;
    int64_t max_slab = 0;                // largest per-chunk code slab (bytes)
    int max_tasks = 0;                   // most warp tasks in one chunk
    int max_spread = 0;                  // largest length difference inside one task
    std::vector<int4> tasks;             // (longest, start in meta, count <= 32, slab byte offset);
                                         // longest | 0x100 when all are that long
    std::vector<int4> chunks;            // (first task, tasks, slab byte offset, slab bytes)
    int64_t slab_bytes = 0;
    OwnedBuf d_plan;                     // chunks, then tasks
    OwnedBuf d_meta;                     // per slot: column in the chunk | length << 16
    OwnedBuf d_slab;                     // per task: longest rows of 32 bytes (4*code per lane)
    Made made;
};

// Queries (rows [r0, r1) of the set; r1 = -1 for all) sorted by length (stable); each length's
// queries fill quads and its quads fill slices.  Empty slots are computed and never stored.
void build_query_plan(QueryPlan& plan, const st_seqset_s& q, cudaStream_t stream, int64_t r0 = 0,
                      int64_t r1 = -1) {
    const int64_t N = (r1 < 0 ? q.count : r1) - r0;
    std::vector<int32_t> order(static_cast<size_t>(N));
    std::vector<int64_t> at(size_t(q.max_len) + 2, 0);
    for (int64_t i = 0; i < N; ++i) at[size_t(q.h_len[size_t(r0 + i)]) + 1]++;
    for (size_t l = 1; l < at.size(); ++l) at[l] += at[l - 1];
    for (int64_t i = 0; i < N; ++i) order[size_t(at[size_t(q.h_len[size_t(r0 + i)])]++)] = int32_t(r0 + i);
    plan.quads.clear();
    plan.slices.clear();
    plan.prof_rows = 0;
    for (int64_t i = 0; i < N;) {
        const int32_t m = q.h_len[size_t(order[size_t(i)])];
        int64_t e = i;
        while (e < N && q.h_len[size_t(order[size_t(e)])] == m) ++e;
        for (int64_t t = i; t < e; t += kSliceQ) {
            const int first = int(plan.quads.size());
            for (int64_t u = t; u < std::min<int64_t>(e, t + kSliceQ); u += 4) {
                int v[4];
                for (int x = 0; x < 4; ++x) v[x] = u + x < e ? order[size_t(u + x)] : -1;
                plan.quads.push_back(make_int4(v[0], v[1], v[2], v[3]));
            }
            plan.slices.push_back(
                make_int4(first, int(plan.quads.size()) - first, m, int(plan.prof_rows)));
            plan.prof_rows += m;
        }
        i = e;
    }
    if (plan.prof_rows > INT32_MAX) fail(ST_EINVAL, "seqtree_b200: query set too large for one call");
    std::vector<int4> up(plan.quads);
    up.insert(up.end(), plan.slices.begin(), plan.slices.end());
    h2d(plan.d_plan.as<int4>(up.size(), stream), up.data(), sizeof(int4) * up.size(), stream);
    for (auto& p : plan.profiles) p->key.clear();
    if (q.owns && r1 < 0) plan.made.on(stream);
    plan.uid = q.uid;
    plan.r0 = r0;
    plan.r1 = r1;
}

// Refs in chunks of rc columns (original order), sorted by length inside a chunk and taken 32 at a
// time (fewer at the end of the chunk, and where lengths would differ by more than kMaxSpread): the
// warp tasks, which follow from the chunk's length histogram alone.  The order inside a length is
// chunk_order_kernel's.  Each task's code rows occupy longest * 32 bytes of the slab, so a chunk's
// slab is one contiguous range.
void build_ref_plan(RefPlan& plan, const st_seqset_s& r, int rc) {
    const int64_t K = r.count;
    plan.rc = rc;
    plan.nchunks = ceil_div(K, rc);
    plan.tasks.clear();
    plan.chunks.clear();
    plan.max_slab = 0;
    plan.max_tasks = 0;
    plan.max_spread = 0;
    std::vector<int32_t> hist(size_t(r.max_len) + 1);
    int64_t slab = 0;
    for (int64_t c = 0; c < plan.nchunks; ++c) {
        const int64_t k0 = c * rc, k1 = std::min<int64_t>(K, k0 + rc);
        std::fill(hist.begin(), hist.end(), 0);
        for (int64_t k = k0; k < k1; ++k) hist[size_t(r.h_len[size_t(k)])]++;
        const int64_t slab0 = slab;
        const int first_task = int(plan.tasks.size());
        int shortest = 0, longest = 0, count = 0;
        int64_t start = k0;
        auto close = [&] {
            if (!count) return;
            plan.max_spread = std::max(plan.max_spread, longest - shortest);
            plan.tasks.push_back(make_int4(longest | (longest == shortest ? 0x100 : 0), int32_t(start),
                                           count, int32_t(slab)));
            slab += int64_t(longest) * 32;
            start += count;
            count = 0;
        };
        for (int l = 0; l <= r.max_len; ++l) {
            int left = hist[size_t(l)];
            if (left && count && l - shortest > kMaxSpread) close();
            while (left) {
                if (!count) shortest = l;
                longest = l;
                const int take = std::min(left, 32 - count);
                count += take;
                left -= take;
                if (count == 32) close();
            }
        }
        close();
        plan.max_slab = std::max(plan.max_slab, slab - slab0);
        const int ntasks = int(plan.tasks.size()) - first_task;
        plan.max_tasks = std::max(plan.max_tasks, ntasks);
        plan.chunks.push_back(make_int4(first_task, ntasks, int(slab0), int(slab - slab0)));
        if (slab > INT32_MAX) fail(ST_EINVAL, "seqtree_b200: reference set too large for one call");
    }
    plan.ntasks = int64_t(plan.tasks.size());
    plan.slab_bytes = slab;
}

// A resident ref set's plans, one per chunk width.
struct RefPlans {
    std::vector<std::unique_ptr<RefPlan>> of;
};

template <class Plan>
Plan& plan_slot(std::shared_ptr<void>& own, std::shared_ptr<void>& shared, bool owns) {
    std::shared_ptr<void>& slot = owns ? own : shared;
    if (!slot) slot = std::make_shared<Plan>();
    return *static_cast<Plan*>(slot.get());
}

// The slices' profiles, one block per slice: word (row j, quad, b) holds pen(q[j], b) of the
// quad's four queries, 8 bits each; WIDE rows hold two words per quad and residue, [quad][half][32]
// with queries 0 | 2 << 16 in half 0 and 1 | 3 << 16 in half 1.  Zero beyond A; empty slots hold the
// largest penalty, so that the sparse sweep's early end does not wait for them.
template <bool WIDE>
__global__ void profile_kernel(const uint8_t* __restrict__ codes, const int64_t* __restrict__ off,
                               const int4* __restrict__ quads, const int4* __restrict__ slices,
                               const int32_t* __restrict__ pen, int A, uint32_t maxpen,
                               uint32_t* __restrict__ prof) {
    const int4 sl = slices[blockIdx.x];
    constexpr int kWords = kQuads * kRow * (WIDE ? 2 : 1);
    uint32_t* dst = prof + int64_t(sl.w) * kWords;
    for (int i = threadIdx.x; i < sl.z * kWords; i += blockDim.x) {
        const int j = i / kWords, w = i - j * kWords;
        const int quad = w / (kWords / kQuads), half = (w / kRow) & 1, b = w & (kRow - 1);
        uint32_t v = 0;
        if (b < A) {
            const int4 q = quad < sl.y ? quads[sl.x + quad] : make_int4(-1, -1, -1, -1);
            const int qs[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                if (WIDE && (x & 1) != half) continue;
                const uint32_t p =
                    qs[x] < 0 ? maxpen : uint32_t(pen[int(codes[off[qs[x]] + j]) * A + b]);
                v |= p << (WIDE ? 16 * (x >> 1) : 8 * x);
            }
        }
        dst[i] = v;
    }
}

// A task's code rows j0, j0 + step, ...: 32 lane bytes each, 4*code of the lane's ref (the null code
// past a ref's end and past the task's count).
__device__ __forceinline__ void fill_task(const uint8_t* codes, const int64_t* off, const uint32_t* meta, int4 t,
                                          int rc, int lane, int j0, int step, uint8_t* slab) {
    const int rows = t.x & 0xFF;
    const uint32_t mt = lane < t.z ? meta[t.y + lane] : 0u;
    const int n = int(mt >> 16);
    const uint8_t* src = codes + (lane < t.z ? off[int64_t(t.y) / rc * rc + (mt & 0xFFFFu)] : 0);
#pragma unroll 4
    for (int j = j0; j < rows; j += step)
        slab[int64_t(t.w) + j * 32 + lane] = uint8_t((j < n ? int(src[j]) : kNullCode) * 4);
}

// Slots of one chunk (one block): its columns sorted by length, and inside a length so that
// neighbours have different columns modulo 32 -- each round takes one ref of every residue -- which
// puts the dense tile's words of a task into different banks.  (Which of several refs of one
// length and residue comes first does not matter.)
constexpr int kMaxRounds = 40;  // rc / 32 of the widest chunk

// With SLAB the block goes on to write its chunk's code slab (a launch less, for few chunks).
template <bool SLAB>
__global__ void __launch_bounds__(256) chunk_order_kernel(const int32_t* __restrict__ rlen, int64_t K, int rc,
                                                          int max_len, uint32_t* __restrict__ meta,
                                                          const uint8_t* __restrict__ codes,
                                                          const int64_t* __restrict__ off,
                                                          const int4* __restrict__ chunks,
                                                          const int4* __restrict__ tasks,
                                                          uint8_t* __restrict__ slab) {
    __shared__ uint32_t occ[65 * 32];
    __shared__ uint32_t at[65 * kMaxRounds];
    const int64_t k0 = int64_t(blockIdx.x) * rc;
    const int kcount = int(K - k0 < rc ? K - k0 : rc);
    const int rounds = rc / 32, buckets = (max_len + 1) * rounds;
    for (int i = threadIdx.x; i < (max_len + 1) * 32; i += 256) occ[i] = 0u;
    for (int i = threadIdx.x; i < buckets; i += 256) at[i] = 0u;
    __syncthreads();
    uint32_t bucket[kMaxRounds * 32 / 256];
#pragma unroll
    for (int t = 0; t < kMaxRounds * 32 / 256; ++t) {
        const int c = t * 256 + threadIdx.x;
        if (c < kcount) {
            const int l = rlen[k0 + c];
            bucket[t] = uint32_t(l) * rounds + atomicAdd(&occ[l * 32 + (c & 31)], 1u);
            atomicAdd(&at[bucket[t]], 1u);
        }
    }
    __syncthreads();
    if (threadIdx.x < 32) {  // exclusive prefix of the buckets by one warp
        uint32_t base = 0;
        for (int b0 = 0; b0 < buckets; b0 += 32) {
            const int b = b0 + int(threadIdx.x);
            const uint32_t v = b < buckets ? at[b] : 0u;
            uint32_t incl = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
                if (int(threadIdx.x) >= o) incl += u;
            }
            if (b < buckets) at[b] = base + incl - v;
            base += __shfl_sync(0xffffffffu, incl, 31);
        }
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < kMaxRounds * 32 / 256; ++t) {
        const int c = t * 256 + threadIdx.x;
        if (c < kcount)
            meta[k0 + atomicAdd(&at[bucket[t]], 1u)] = uint32_t(c) | (bucket[t] / rounds) << 16;
    }
    if constexpr (SLAB) {
        __syncthreads();  // also makes the block's global writes visible to the block
        const int4 ch = chunks[blockIdx.x];
        for (int u = threadIdx.x >> 5; u < ch.y; u += 8)
            fill_task(codes, off, meta, tasks[ch.x + u], rc, threadIdx.x & 31, 0, 1, slab);
    }
}

__global__ void ref_slab_kernel(const uint8_t* __restrict__ codes, const int64_t* __restrict__ off,
                                const uint32_t* __restrict__ meta, const int4* __restrict__ tasks, int rc,
                                uint8_t* __restrict__ slab) {
    fill_task(codes, off, meta, tasks[blockIdx.x], rc, threadIdx.x & 31, threadIdx.x >> 5, blockDim.x >> 5,
              slab);
}

// ---------------------------------------------------------------------------- fast kernel ---
// Shared memory of one CTA: byte offsets, in this order.
struct FastSmem {
    int codes, tile, bits, frow, task, meta, bar, total;
};

struct FastArgs {
    const uint32_t* prof;
    const uint8_t* slab;     // ref code slab
    const int32_t* rlen;
    int64_t K;
    int rc;                  // columns per chunk
    const int4* quads;       // original query indices; -1 marks an empty slot
    const int4* slices;      // (first quad, quads, length, profile row offset)
    int64_t nslices;
    const uint32_t* ref_meta;  // per sorted slot: column in the chunk | length << 16
    const int4* tasks;
    const int4* chunks;      // (first task, tasks, slab byte offset, slab bytes)
    FastSmem sm;
    int score16;             // sparse sums of 16 bits (else 8: no hit's sum is above 255)
    int spread;              // rows past the query that a mixed task's diagonal may read
    const uint32_t* prior2;  // rows (M*W1 + d) of pstride words: [3] the first value, [4 + j] steps
    int pstride;
    const int32_t* ftab;     // [m*W1 + n]: per-(m,n) additive term (prior minimum + gap cost)
    int W1;
    int32_t* out;            // dense output (unused by the sparse form)
    unsigned long long* err; // set when the bounded wait for the staging copies gives up
    SparseSink sink;         // sparse output (unused by the dense form)
};

// One non-blocking probe of an mbarrier phase (callers bound the number of probes).
__device__ __forceinline__ uint32_t mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok;
}

__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes,
                                         uint32_t bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"(dst),
        "l"(src), "r"(bytes), "r"(bar)
        : "memory");
}

inline FastSmem fast_smem(int prof_cap, int slab_cap, int rc, int W1, int max_tasks, int score_bytes) {
    FastSmem m;
    auto up = [](int v) { return (v + 15) & ~15; };
    m.codes = prof_cap;
    m.tile = m.codes + up(slab_cap);
    // prof_cap: a slice's profile and its zero rows; slab_cap: a chunk's code slab; the tile is rc
    // columns of kTileW words (dense, score_bytes 0), or scores [query][column] and the hit bitmap
    m.bits = m.tile + up(score_bytes ? kSliceQ * rc * score_bytes : rc * kTileW * 4);
    m.frow = m.bits + up(score_bytes ? kSliceQ * (rc / 32) * 4 : 0);
    m.task = m.frow + up(W1 * 4);
    m.meta = m.task + up(max_tasks * 16);
    m.bar = m.meta + up(rc * 4);
    m.total = m.bar + 16;
    return m;
}

// The (even, odd) int16x2 words of a quad at one profile address.
template <bool WIDE>
__device__ __forceinline__ void quad_words(const uint8_t* p, uint32_t& e, uint32_t& o) {
    if constexpr (WIDE) {
        e = *reinterpret_cast<const uint32_t*>(p);
        o = *reinterpret_cast<const uint32_t*>(p + kRow * 4);
    } else {
        const uint32_t w = *reinterpret_cast<const uint32_t*>(p);
        o = __byte_perm(w, 0u, 0x4341);  // bytes 1 and 3
        e = w - o * 256u;                // bytes 0 and 2, an IMAD
    }
}

// One warp unit: NQ quads of the slice against the 32 refs of one task.  Per position: one or two
// code bytes, 2 * NQ lookups at immediates from two addresses, and per quad two splits, two adds and
// two DPX minima.  What bounds it: issue slots (10 per quad and position, 2.5 cycles of an SM's
// four schedulers), with the LDS pipe (2 cycles), the ALU (2 to 3) and the FMA pipe just below.
// SPARSE without a prior: both states only grow, so once every A and B of the warp is above its
// lane's threshold no cell can pass and the unit ends (false).  Looked at every four positions from
// the eighth on: 13 instructions, against 44 a position; on junctions with BLOSUM62 at 24 the
// sweep ends after 9.8 of 13.2 positions on average.
template <int NQ, bool PRIOR, bool WIDE, bool SPARSE>
__device__ __forceinline__ bool run_unit(const FastArgs& a, const uint8_t* s_prof, const uint8_t* rows0,
                                         int m, int n, int nmax, bool same_len, uint32_t lim,
                                         uint32_t (&res)[2 * NQ]) {
    constexpr bool kStop = SPARSE && !PRIOR;
    constexpr int kQuadB = kRow * 4 * (WIDE ? 2 : 1);
    constexpr int kRowB = kQuadB * kQuads;
    const int L = min(m, nmax);
    if (same_len && nmax == m) {  // no block: the plain sum
#pragma unroll
        for (int q = 0; q < 2 * NQ; ++q) res[q] = 0u;
        auto step = [&](int j) {
            const uint8_t* p = s_prof + j * kRowB + rows0[j * 32];
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                uint32_t e, o;
                quad_words<WIDE>(p + q * kQuadB, e, o);
                res[2 * q] += e;
                res[2 * q + 1] += o;
            }
        };
        int j = 0;
        for (; j + 4 <= L; j += 4) {
            if (kStop && j >= 8) {
                uint32_t low = res[0];
#pragma unroll
                for (int q = 1; q < 2 * NQ; q += 2)
                    low = __vimin3_s16x2(low, res[q], q + 1 < 2 * NQ ? res[q + 1] : res[q]);
                if (!__any_sync(0xffffffffu, (lim - low) & 0x80008000u)) return false;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) step(j + u);
        }
        for (; j < L; ++j) step(j);
        return true;
    }
    // Diagonal d: a longer query reads d profile rows further down, a longer ref reads the residue d
    // positions further on.
    const uint8_t* pd = s_prof + max(m - n, 0) * kRowB;
    const uint8_t* rowsd = rows0 + max(n - m, 0) * 32;
    const uint32_t* prow =
        PRIOR ? a.prior2 + (size_t(max(m, n)) * a.W1 + abs(m - n)) * a.pstride : nullptr;
    uint32_t A[2 * NQ];
    const uint32_t first = PRIOR ? __ldg(prow + 3) : 0u;
#pragma unroll
    for (int q = 0; q < 2 * NQ; ++q) A[q] = res[q] = first;
    // The sweep, in two versions: when no ref is longer than the query both diagonals read
    // residue j of the ref, so one byte load serves both addresses.
    auto sweep = [&](auto same_residue) {
        constexpr bool kSame = decltype(same_residue)::value;
        auto step = [&](int j, uint32_t dp) {
            const uint32_t c0 = rows0[j * 32];
            const uint8_t* p0 = s_prof + j * kRowB + c0;
            const uint8_t* p1 = pd + j * kRowB + (kSame ? c0 : uint32_t(rowsd[j * 32]));
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                uint32_t e0, o0, e1, o1;
                quad_words<WIDE>(p0 + q * kQuadB, e0, o0);
                quad_words<WIDE>(p1 + q * kQuadB, e1, o1);
                A[2 * q] += PRIOR ? e0 + dp : e0;
                A[2 * q + 1] += PRIOR ? o0 + dp : o0;
                res[2 * q] = __viaddmin_s16x2(res[2 * q], e1, A[2 * q]);
                res[2 * q + 1] = __viaddmin_s16x2(res[2 * q + 1], o1, A[2 * q + 1]);
            }
        };
        // The prior's steps of the next group of four positions are requested one group ahead,
        // so their load latency hides behind the current group's lookups.
        int j = 0;
        uint4 pnext = make_uint4(0u, 0u, 0u, 0u);
        if constexpr (PRIOR)
            if (L >= 4) pnext = __ldg(reinterpret_cast<const uint4*>(prow + 4));
        for (; j + 4 <= L; j += 4) {
            if (kStop && j >= 8) {
                uint32_t low = __vimin3_s16x2(A[0], res[0], res[1]);
#pragma unroll
                for (int q = 1; q < 2 * NQ; ++q)
                    low = __vimin3_s16x2(low, A[q], q + 1 < 2 * NQ ? res[q + 1] : A[q]);
                if (!__any_sync(0xffffffffu, (lim - low) & 0x80008000u)) return false;
            }
            const uint4 pv = pnext;
            if constexpr (PRIOR)
                if (j + 8 <= L) pnext = __ldg(reinterpret_cast<const uint4*>(prow + j + 8));
            step(j, pv.x);
            step(j + 1, pv.y);
            step(j + 2, pv.z);
            step(j + 3, pv.w);
        }
        for (; j < L; ++j) step(j, PRIOR ? __ldg(prow + j + 4) : 0u);
        return true;
    };
    return nmax <= m ? sweep(std::true_type{}) : sweep(std::false_type{});
}

// One CTA per (chunk, slice).  CTAs per SM: three of 80 registers, or in the sparse form four of 64,
// which with 8-bit scores fit at the 1,024-column width: 148 -> 139 ms on 100,000 x 1,000,000 (a
// tile's staging and its barriers are then covered by three others).  Narrower chunks
// cost more tiles: 3.0 (1,024) / 3.3 (768) / 3.8 (512) / 5.1 ms (256) per 2e9 pairs.
// WRAPS: the sparse form where some sum + term may pass the end of int32 (a test of its own on every
// hit costs 7 % where 2.75 % of the cells are hits, so it is a variant).
template <bool PRIOR, bool WIDE, bool SPARSE, bool WRAPS = false>
__global__ void __launch_bounds__(kThreads, SPARSE ? 4 : 3) gapblock_fast_kernel(const FastArgs a) {
    extern __shared__ __align__(128) uint8_t smem[];
    const FastSmem& sm = a.sm;
    constexpr int kRowB = kRow * 4 * kQuads * (WIDE ? 2 : 1);
    uint8_t* s_codes = smem + sm.codes;
    uint32_t* s_tile = reinterpret_cast<uint32_t*>(smem + sm.tile);
    uint8_t* s_score = smem + sm.tile;
    uint32_t* s_bits = reinterpret_cast<uint32_t*>(smem + sm.bits);
    int32_t* s_frow = reinterpret_cast<int32_t*>(smem + sm.frow);
    int4* s_task = reinterpret_cast<int4*>(smem + sm.task);
    uint32_t* s_meta = reinterpret_cast<uint32_t*>(smem + sm.meta);
    uint64_t* s_bar = reinterpret_cast<uint64_t*>(smem + sm.bar);

    const int64_t slice = blockIdx.y + int64_t(blockIdx.z) * gridDim.y;  // slices past 65,535 use z
    if (slice >= a.nslices) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t bar = uint32_t(__cvta_generic_to_shared(s_bar));
    const int chunk = blockIdx.x;
    const int64_t k0 = int64_t(chunk) * a.rc;
    const int kcount = int(a.K - k0 < a.rc ? a.K - k0 : a.rc);
    const int4 sl = a.slices[slice];
    const int nq = sl.y, m = sl.z;
    const int4 ch = a.chunks[chunk];
    const int t0 = ch.x, nt = ch.y, slab0 = ch.z, slab_bytes = ch.w;

    // Stage the slice's profile and the chunk's code slab with two bulk (TMA) copies that complete
    // on one mbarrier, while the threads load the rest.
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar));
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                     "r"(uint32_t(m * kRowB + slab_bytes))
                     : "memory");
        if (m > 0)
            bulk_g2s(uint32_t(__cvta_generic_to_shared(smem)),
                     reinterpret_cast<const uint8_t*>(a.prof) + int64_t(sl.w) * kRowB,
                     uint32_t(m * kRowB), bar);
        if (slab_bytes > 0)
            bulk_g2s(uint32_t(__cvta_generic_to_shared(s_codes)), a.slab + slab0,
                     uint32_t(slab_bytes), bar);
    }
    // Per-tile metadata: the (m, n) terms, the chunk's tasks, each sorted slot's column and length.
    // Rows past the query keep the null column at 0 for lanes past their ref's end.
    // The sparse form keeps the test word instead of the term: 0x8000 + T in both halves, T =
    // threshold - term; a half is a hit when it is at most T, bit 15 of the difference.  Beside a term
    // so near the end of int32 that the score may wrap below 0, every half is tested again as a score.
    for (int i = tid; i < a.W1; i += kThreads) {
        const int32_t f = a.ftab[m * a.W1 + i];
        const int64_t room = WRAPS && f > INT32_MAX - kMaxHalf ? kMaxHalf : int64_t(a.sink.thresh) - f;
        s_frow[i] = !SPARSE ? f
                    : room >= 0 ? int32_t(0x80008000u + uint32_t(room < kMaxHalf ? room : kMaxHalf) * 0x10001u)
                                : 0x7FFF7FFF;
    }
    for (int i = tid; i < a.spread * kQuads * (WIDE ? 2 : 1); i += kThreads)
        reinterpret_cast<uint32_t*>(smem + m * kRowB)[i * kRow + kNullCode] = 0u;
#pragma unroll 4
    for (int c = tid; c < kcount; c += kThreads) s_meta[c] = a.ref_meta[k0 + c];
    if (SPARSE)
        for (int i = tid; i < kSliceQ * (a.rc / 32) / 4; i += kThreads)
            reinterpret_cast<uint4*>(s_bits)[i] = make_uint4(0u, 0u, 0u, 0u);
    for (int i = tid; i < nt; i += kThreads) s_task[i] = a.tasks[t0 + i];
    __syncthreads();
    {
        // Bounded wait on phase 0 by every thread.  If any thread runs out, the CTA records
        // the failure, waits once more (bounded) for its copies in flight, and leaves as a
        // whole -- the host then reports ST_ETIMEOUT and no tile is stored.
        uint32_t done = 0;
        for (int it = 0; it < (1 << 20) && !done; ++it) done = mbar_try_wait(bar, 0);
        if (__syncthreads_or(!done)) {
            if (tid == 0) atomicExch(a.err, 1ull);
            for (int it = 0; it < (1 << 20) && !done; ++it) done = mbar_try_wait(bar, 0);
            __syncthreads();
            return;
        }
    }

    for (int t = warp; t < nt; t += kWarps) {
        const int4 task = s_task[t];
        const int nmax = task.x & 0xFF;
        const bool same_len = (task.x & 0x100) != 0;
        const bool live = lane < task.z;
        const uint32_t meta = s_meta[int(task.y - k0) + (live ? lane : 0)];
        const int n = live ? int(meta >> 16) : nmax;
        const int col = int(meta & 0xFFFFu);
        const uint8_t* rows0 = s_codes + (task.w - slab0) + lane;
        const int32_t f = s_frow[n];
        const uint32_t lim = live ? uint32_t(f) : 0x7FFF7FFFu;
        auto unit = [&](auto quads) {
            constexpr int NQ = decltype(quads)::value;
            uint32_t res[2 * NQ];
            const bool done =
                run_unit<NQ, PRIOR, WIDE, SPARSE>(a, smem, rows0, m, n, nmax, same_len, lim, res);
            if constexpr (!SPARSE) {
                if (live) {
                    uint32_t* dst = s_tile + col * kTileW;
#pragma unroll
                    for (int q = 0; q < 2 * NQ; ++q) dst[q] = res[q];
                    dst[2 * kQuads] = uint32_t(f);
                }
            } else {
                if (!done) return;
                uint32_t any = 0u;
#pragma unroll
                for (int q = 0; q < 2 * NQ; ++q) any |= lim - res[q];
                if (any & 0x80008000u) {
#pragma unroll
                    for (int q = 0; q < 2 * NQ; ++q) {
                        const uint32_t hit = lim - res[q];
                        // word q of quad q / 2: queries (q & 1) and (q & 1) + 2
                        const int row = (q >> 1) * 4 + (q & 1);
                        auto keep = [&](int at, uint32_t v) {
                            if (WRAPS && int32_t((v & 0xFFFFu) + uint32_t(__ldg(a.ftab + m * a.W1 + n))) > a.sink.thresh)
                                return;
                            atomicOr(s_bits + at * (a.rc / 32) + (col >> 5), 1u << (col & 31));
                            if (a.score16)
                                reinterpret_cast<uint16_t*>(s_score)[at * a.rc + col] = uint16_t(v);
                            else
                                s_score[at * a.rc + col] = uint8_t(v);
                        };
                        if (hit & 0x8000u) keep(row, res[q]);
                        if (hit & 0x80000000u) keep(row + 2, res[q] >> 16);
                    }
                }
            }
        };
        if (nq > 2)
            unit(std::integral_constant<int, 4>{});
        else if (nq == 2)
            unit(std::integral_constant<int, 2>{});
        else
            unit(std::integral_constant<int, 1>{});
    }
    __syncthreads();

    if constexpr (!SPARSE) {
        // Warp w writes the two rows of result word w: 128 contiguous bytes per store.
        const int quad = warp >> 1;
        if (quad < nq) {
            const int4 q = a.quads[sl.x + quad];
            const int q1 = (warp & 1) ? q.y : q.x, q2 = (warp & 1) ? q.w : q.z;
            int32_t* d1 = a.out + int64_t(q1) * a.K + k0;
            int32_t* d2 = a.out + int64_t(q2) * a.K + k0;
#pragma unroll 4
            for (int c = lane; c < kcount; c += 32) {
                const uint32_t v = s_tile[c * kTileW + warp], f = s_tile[c * kTileW + 2 * kQuads];
                if (q1 >= 0) d1[c] = int32_t((v & 0xFFFFu) + f);
                if (q2 >= 0) d2[c] = int32_t((v >> 16) + f);
            }
        }
    } else {
        // Warp w owns queries 2w and 2w + 1 of the slice: it counts their hits, reserves a segment
        // for them and writes each row's hits there in ascending column order, recording the piece
        // (row, chunk) it wrote.  (One reservation per CTA made every warp wait for the atomic's
        // round trip on each tile.)
        const unsigned full = 0xffffffffu;
        const int words = (kcount + 31) >> 5, pitch = a.rc / 32;
        if ((warp >> 1) >= nq) return;
        const int4 q = a.quads[sl.x + (warp >> 1)];
        const int qrow[2] = {(warp & 1) ? q.z : q.x, (warp & 1) ? q.w : q.y};
        int cnt[2] = {0, 0};
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            if (qrow[r] < 0) continue;
            int n = 0;
            for (int w = lane; w < words; w += 32) n += __popc(s_bits[(warp * 2 + r) * pitch + w]);
            cnt[r] = int(__reduce_add_sync(full, unsigned(n)));
        }
        const int tot = cnt[0] + cnt[1];
        unsigned long long off = 0;
        if (tot > 0) {
            if (lane == 0) off = atomicAdd(a.sink.count, (unsigned long long)tot);
            off = __shfl_sync(full, off, 0);
        }
        const bool fits = off + tot <= a.sink.cap;  // else counted only; the host re-runs
        const int row_of = lane ? qrow[1] : qrow[0];
        if (lane < 2 && row_of >= 0) {
            const int64_t piece = (int64_t(row_of) - a.sink.row0) * a.sink.nchunks + chunk;
            a.sink.piece_cnt[piece] = lane ? cnt[1] : cnt[0];
            if (tot > 0) a.sink.piece_off[piece] = int64_t(off + (lane ? cnt[0] : 0));
        }
        if (tot == 0 || !fits) return;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            if (cnt[r] == 0) continue;
            const int row = warp * 2 + r;
            for (int w0 = 0; w0 < words; w0 += 32) {
                uint32_t word = w0 + lane < words ? s_bits[row * pitch + w0 + lane] : 0u;
                const int c0 = __popc(word);
                int incl = c0;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(full, incl, o);
                    if (lane >= o) incl += t;
                }
                unsigned long long pos = off + (unsigned long long)(incl - c0);
                while (word) {
                    const int c = (w0 + lane) * 32 + __ffs(int(word)) - 1;
                    word &= word - 1;
                    const int at = row * a.rc + c;
                    const uint32_t v = a.score16 ? reinterpret_cast<const uint16_t*>(s_score)[at] : s_score[at];
                    a.sink.seg[pos++] = make_int2(
                        int(k0 + c), int(v + uint32_t(__ldg(a.ftab + m * a.W1 + a.rlen[k0 + c]))));
                }
                off += (unsigned long long)__shfl_sync(full, incl, 31);
            }
        }
    }
}

// ---------------------------------------------------------------------------- general -------
struct GeneralArgs {
    const uint8_t* qcodes;
    const int64_t* qoff;
    const uint8_t* rcodes;
    const int64_t* roff;
    int64_t row0;         // first query row (row blocks of the sparse form)
    int64_t N, K;         // rows in this launch, refs
    const int32_t* pen;   // A*A
    int A;
    int32_t go, ge;
    const int32_t* prior; // (pw+1)^3 or null
    int64_t pw1;
    int32_t* out;         // dense output (unused by the sparse form)
    SparseSink sink;      // sparse output (unused by the dense form)
};

// The gap-block score of one pair in int32 arithmetic with the reference's wrap
// (src/gapblock.cpp:39-62, in the single-sweep form S + min_i(C_i + p_i)).
// Score of one pair; with `pos`, also the block position of the minimum (the smallest such
// position; 0 when the lengths are equal), counted in residues of the shorter sequence.
__device__ __forceinline__ int32_t gapblock_cell(const uint8_t* q, int m, const uint8_t* r, int n,
                                                 const int32_t* s_pen, int A, int32_t go, int32_t ge,
                                                 const int32_t* prior, int64_t pw1,
                                                 int32_t* pos = nullptr) {
    const int L = min(m, n), d = abs(m - n);
    if (pos) *pos = 0;
    if (d == 0) {
        uint32_t s = 0;
        for (int j = 0; j < L; ++j) s += uint32_t(s_pen[q[j] * A + r[j]]);
        return int32_t(s);
    }
    const bool ql = m > n;
    const int32_t* prow = prior ? prior + (int64_t(max(m, n)) * pw1 + d) * pw1 : nullptr;
    int32_t S = 0, C = 0;
    int32_t best = prow ? prow[0] : 0;
    int32_t at = 0;
    for (int j = 0; j < L; ++j) {
        const int32_t p0v = s_pen[q[j] * A + r[j]];
        const int32_t pdv = ql ? s_pen[q[j + d] * A + r[j]] : s_pen[q[j] * A + r[j + d]];
        S += pdv;
        C += p0v - pdv;
        const int32_t cand = C + (prow ? prow[j + 1] : 0);
        if (cand < best) {
            best = cand;
            at = j + 1;
        }
    }
    if (pos) *pos = at;
    return int32_t(uint32_t(S) + uint32_t(best) + uint32_t(go) + uint32_t(d - 1) * uint32_t(ge));
}

// One thread per listed pair (qi[p], ri[p]); out[p] = its score.
__global__ void __launch_bounds__(256) gapblock_pairs_kernel(
    const uint8_t* __restrict__ qcodes, const int64_t* __restrict__ qoff,
    const uint8_t* __restrict__ rcodes, const int64_t* __restrict__ roff,
    const int32_t* __restrict__ qi, const int32_t* __restrict__ ri, int64_t n,
    const int32_t* __restrict__ pen, int A, int32_t go, int32_t ge,
    const int32_t* __restrict__ prior, int64_t pw1, int32_t* __restrict__ out,
    int32_t* __restrict__ pos_out) {
    extern __shared__ int32_t s_pen[];
    for (int i = threadIdx.x; i < A * A; i += blockDim.x) s_pen[i] = pen[i];
    __syncthreads();
    for (int64_t p = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; p < n;
         p += int64_t(gridDim.x) * blockDim.x) {
        const int64_t i = qi[p], k = ri[p];
        const int m = int(qoff[i + 1] - qoff[i]), nn = int(roff[k + 1] - roff[k]);
        int32_t at = 0;
        out[p] = gapblock_cell(qcodes + qoff[i], m, rcodes + roff[k], nn, s_pen, A, go, ge, prior,
                               pw1, pos_out ? &at : nullptr);
        if (pos_out) pos_out[p] = at;
    }
}

// One thread per (i, k) in row-major order, int32 arithmetic with the reference's wrap.  The
// loop runs the same number of rounds on every lane (the sparse append is warp-collective).
template <bool SPARSE>
__global__ void __launch_bounds__(256) gapblock_general_kernel(const GeneralArgs a) {
    extern __shared__ int32_t s_pen[];
    for (int i = threadIdx.x; i < a.A * a.A; i += blockDim.x) s_pen[i] = a.pen[i];
    __syncthreads();
    const int64_t total = a.N * a.K;
    for (int64_t base = int64_t(blockIdx.x) * blockDim.x; base < total;
         base += int64_t(gridDim.x) * blockDim.x) {
        const int64_t idx = base + threadIdx.x;
        if (!SPARSE && idx >= total) break;
        const bool live = idx < total;
        const int64_t il = live ? idx / a.K : 0, k = live ? idx - il * a.K : 0;
        const int64_t i = a.row0 + il;
        const int m = int(a.qoff[i + 1] - a.qoff[i]);
        const int n = int(a.roff[k + 1] - a.roff[k]);
        const int32_t v = gapblock_cell(a.qcodes + a.qoff[i], m, a.rcodes + a.roff[k], n, s_pen,
                                        a.A, a.go, a.ge, a.prior, a.pw1);
        if constexpr (SPARSE) {
            sink_append(a.sink, live && v <= a.sink.thresh ? 1u : 0u, int(threadIdx.x & 31),
                        [&](int, unsigned long long& key, int32_t& val) {
                            key = sink_key(a.sink, i, k);
                            val = v;
                        });
        } else {
            a.out[idx] = v;
        }
    }
}

using FastKernel = void (*)(FastArgs);

template <bool SPARSE, bool WRAPS>
FastKernel fast_kernel(bool prior, bool wide) {
    return prior ? (wide ? gapblock_fast_kernel<true, true, SPARSE, WRAPS> : gapblock_fast_kernel<true, false, SPARSE, WRAPS>)
                 : (wide ? gapblock_fast_kernel<false, true, SPARSE, WRAPS> : gapblock_fast_kernel<false, false, SPARSE, WRAPS>);
}

// Words per prior row: the first value at 3, step j at 4 + j, rounded up so that every row is
// 16-byte aligned and the last aligned group of four stays inside the row.
int prior_stride(int W1) { return (W1 + 3 + 4 + 3) & ~3; }

// Device-side tables of the fast path and the arguments they were built from.  The first 64 argument sets
// of a device (each of at most 1.2 MB, 0.1 with sequences up to 25) are kept and never written again, so
// calls on other streams and captured graphs may read them.  Further ones share one more, as with
// the profiles.
struct GbTables {
    std::vector<uint8_t> key;
    OwnedBuf buf;
    Made made;
    const uint32_t* prior2 = nullptr;
    const int32_t *pen = nullptr, *ftab = nullptr;
    int32_t least_term = 0;  // of ftab: below 0 where a prior's minimum outweighs the gap cost
    int32_t most_term = 0;
};
constexpr size_t kMaxTables = 65;  // the last one changes hands

std::vector<std::unique_ptr<GbTables>>& gb_tables(int device) {
    static std::mutex mu;
    static auto& all = *new std::map<int, std::vector<std::unique_ptr<GbTables>>>;  // (until the process exits)
    std::lock_guard<std::mutex> lk(mu);
    return all[device];
}

// Penalty grid; per-(M,d) prior rows shifted by their minimum (added back through ftab) and
// clamped at CAP = 2 * kMaxSum + 1 -- a clamped position can never win, because the position
// holding the row's minimum scores at most kMaxSum while a clamped one scores above it; a row keeps
// its first value and the steps between values (0 past the last position; A and B stay at most
// kMaxSum + CAP < 2^15, and each packed sum of non-negative halves is exact whatever the step's
// sign).  Nothing here depends on the sets beyond their longest sequence, so calls with new
// queries against the same panel keep the tables;
// ftab[m][n] = prior minimum + gap_open + (d-1)*gap_extend (int32 wrap, as the reference's
// int32 arithmetic).
void build_tables(GbTables& tb, const std::vector<int32_t>& pen, int32_t go, int32_t ge, int W,
                  const int32_t* prior, int64_t W1p, cudaStream_t stream) {
    const int W1 = W + 1;
    constexpr int32_t cap = 2 * kMaxSum + 1;
    std::vector<int32_t> ftab(size_t(W1) * W1, 0);
    const int pstride = prior_stride(W1);
    std::vector<uint32_t> prior2;
    if (prior) prior2.assign(size_t(W1) * W1 * pstride, 0);
    for (int m = 0; m <= W; ++m)
        for (int n = 0; n <= W; ++n) {
            const int M = std::max(m, n), d = std::abs(m - n), L = std::min(m, n);
            if (d == 0) continue;
            int32_t pmin = 0;
            if (prior) {
                const int32_t* row = prior + (int64_t(M) * W1p + d) * W1p;
                pmin = row[0];
                for (int i = 1; i <= L; ++i) pmin = std::min(pmin, row[i]);
                if (m >= n) {  // fill each (M, d) row once
                    uint32_t* dst = prior2.data() + (size_t(M) * W1 + d) * pstride + 3;
                    uint32_t last = 0;
                    for (int i = 0; i <= L; ++i) {
                        const uint32_t v =
                            uint32_t(std::min<int64_t>(int64_t(row[i]) - pmin, cap)) * 0x10001u;
                        dst[i] = v - last;
                        last = v;
                    }
                }
            }
            ftab[size_t(m) * W1 + n] = int32_t(uint32_t(pmin) + uint32_t(go) +
                                               uint32_t(d - 1) * uint32_t(ge));
        }
    tb.least_term = *std::min_element(ftab.begin(), ftab.end());
    tb.most_term = *std::max_element(ftab.begin(), ftab.end());
    // one upload: prior steps (16-byte rows), penalties, terms
    std::vector<uint32_t> up(std::move(prior2));
    const size_t pen_at = up.size(), ftab_at = pen_at + pen.size();
    up.insert(up.end(), pen.begin(), pen.end());
    up.insert(up.end(), ftab.begin(), ftab.end());
    uint32_t* d = tb.buf.as<uint32_t>(up.size(), stream);
    h2d(d, up.data(), up.size() * 4, stream);
    tb.prior2 = d;
    tb.pen = reinterpret_cast<int32_t*>(d + pen_at);
    tb.ftab = reinterpret_cast<int32_t*>(d + ftab_at);
}

// CTAs per SM the fast kernel's registers allow (256 threads of 80 registers, 64 in the sparse form).
constexpr int kTargetBlocks[2] = {3, 4};

int prof_bytes(int max_qlen, int spread, bool wide) {
    return (max_qlen + spread) * kRow * 4 * kQuads * (wide ? 2 : 1);
}

}  // namespace

namespace {

// Chunk widths the fast kernel may use (multiples of 32).  The widest of 1,024 or less that
// reaches the best CTA residency is the static choice; the autotuner measures all of them once per
// shape.
constexpr int kRcCandidates[] = {1280, 1024, 768, 640, 512, 384, 256};
constexpr int kNumRc = int(sizeof(kRcCandidates) / sizeof(kRcCandidates[0]));
static_assert(kRcCandidates[0] <= kMaxRounds * 32, "chunk_order_kernel's buckets");
// Pairs a dense call's first-time tuning runs each variant on (its first query rows).
constexpr int64_t kTuneSlicePairs = int64_t(100) * 1000 * 1000;
thread_local int t_force_rc = 0;      // the chunk width of a run: the tuner's choice, or one it times
thread_local bool t_trial_rc = false;  // (a trial)

// The conditions under which gapblock_run takes the fast kernel (non-negative penalties, every
// length <= 64, halves that cannot carry), the form whose sparse output is ordered.
bool fast_form_possible(const st_seqset_s& qs, const st_seqset_s& rs, const int32_t* penalty,
                        int32_t matrix_size) {
    if (qs.alphabet < 0 || qs.alphabet != rs.alphabet) return false;
    const int A = alphabet_size(qs.alphabet);
    if (penalty && matrix_size != A) return false;
    int64_t maxpen = 0;
    for (int x = 0; x < A; ++x)
        for (int y = 0; y < A; ++y) {
            const int64_t v = penalty ? penalty[x * A + y] : int64_t(x != y);
            if (v < 0) return false;
            maxpen = std::max(maxpen, v);
        }
    const int32_t longest = std::max(qs.max_len, rs.max_len);
    return longest <= 64 && int64_t(std::min(qs.max_len, rs.max_len)) * maxpen <= kMaxSum;
}

std::string gb_shape_key(const st_seqset_s& qs, const st_seqset_s& rs, bool has_prior) {
    return "gapblock|" + std::to_string(qs.max_len) + "|" +
           std::to_string(int(has_prior)) + "|" + std::to_string(std::max(qs.max_len, rs.max_len)) +
           "|" + std::to_string(size_bucket(qs.count)) + "|" + std::to_string(size_bucket(rs.count));
}

// Validated inputs -> the dense matrix in `out_d` (device, N*K int32), or, when `sink` is given,
// the cells that pass its threshold appended to it.
// `r0`, `r1` restrict the queries to rows [r0, r1) (r1 = -1: all rows): the sparse form's row
// blocks, and the dense form's first-time tuning slice (which starts at row 0).
void gapblock_run(st_seqset_s& qs, st_seqset_s& rs, const int32_t* penalty, int32_t matrix_size,
                  int32_t go, int32_t ge, const int32_t* prior, int64_t prior_len,
                  uint32_t prior_width, int32_t* out_d, SparseSink* sink,
                  cudaStream_t stream, int64_t r0 = 0, int64_t r1 = -1) {
    if (go < 0 || ge < 0) fail(ST_EINVAL, "gap_open and gap_extend must be >= 0");
    if (qs.alphabet < 0 || qs.alphabet != rs.alphabet)
        fail(ST_EINVAL, "seqtree_b200: gap-block sets must be encoded with one alphabet");
    const int A = alphabet_size(qs.alphabet);
    if (penalty && matrix_size != A) fail(ST_EINVAL, "matrix size does not match the alphabet");
    const int64_t N = qs.count, K = rs.count;
    if (N == 0 || K == 0) return;
    const int32_t longest = std::max(qs.max_len, rs.max_len);
    const int64_t W1p = int64_t(prior_width) + 1;
    const bool has_prior = prior && prior_len > 0;
    if (has_prior) {
        if (prior_len != W1p * W1p * W1p)
            fail(ST_EINVAL, "prior table must have (prior_width + 1)^3 entries");
        if (uint32_t(longest) > prior_width)
            fail(ST_EINVAL, "a sequence is longer than the prior table's width");
    }
    Context& ctx = context();

    // Penalty grid (unit cost when null): src/gapblock.cpp:25-31.
    std::vector<int32_t> pen(size_t(A) * A);
    for (int x = 0; x < A; ++x)
        for (int y = 0; y < A; ++y) pen[size_t(x) * A + y] = penalty ? penalty[x * A + y] : int32_t(x != y);
    int64_t maxpen = 0;
    bool nonneg = true;
    for (int32_t v : pen) {
        maxpen = std::max<int64_t>(maxpen, v);
        nonneg &= v >= 0;
    }
    const int32_t Lmax = std::min(qs.max_len, rs.max_len);
    const int64_t lmaxpen = int64_t(Lmax) * maxpen;
    bool fast = nonneg && longest <= 64 && lmaxpen <= kMaxSum;

    const int W = longest, W1 = W + 1;
    const bool wide = maxpen > 255;  // the penalties of four queries do not fit one word
    // Tables for this (matrix, gaps, prior, lengths): kept, so repeated calls with the same arguments
    // enqueue nothing but the kernel.
    const StreamNow now(ctx, stream);
    static const GbTables no_tables;  // (the general kernel reads none)
    const GbTables* tbp = &no_tables;
    if (fast) {
        const int64_t hdr[8] = {A, go, ge, W, int64_t(prior_width), has_prior, 0, 0};
        const struct {
            const void* p;
            size_t n;
        } parts[3] = {{hdr, sizeof hdr}, {pen.data(), pen.size() * 4},
                      {prior, has_prior ? size_t(prior_len) * 4 : 0}};
        Phase ph("tables");
        auto same = [&](const GbTables& t) {
            if (t.key.size() != parts[0].n + parts[1].n + parts[2].n) return false;
            size_t at = 0;
            for (const auto& part : parts) {
                if (part.n && std::memcmp(t.key.data() + at, part.p, part.n) != 0) return false;
                at += part.n;
            }
            return true;
        };
        auto& kept = gb_tables(ctx.device);
        static thread_local size_t recent = 0;  // most calls repeat the last one's arguments
        auto it = kept.begin() + int64_t(std::min(recent, kept.size()));
        if (it == kept.end() || !same(**it))
            it = std::find_if(kept.begin(), kept.end(), [&](const auto& t) { return same(*t); });
        recent = size_t(it - kept.begin());
        const bool last = it != kept.end() ? it + 1 == kept.end() && kept.size() == kMaxTables
                                           : kept.size() + 1 >= kMaxTables;
        if (last) refuse_capture(stream);
        if (it != kept.end()) {
            (*it)->made.need(now);
            tbp = it->get();
        } else {
            auto fresh = std::make_unique<GbTables>();
            if (kept.size() == kMaxTables) {
                STB_CUDA(cudaDeviceSynchronize());  // any stream's kernels may read them
                fresh = std::move(kept.back());
                kept.pop_back();
                fresh->key.clear();
            }
            build_tables(*fresh, pen, go, ge, W, has_prior ? prior : nullptr, W1p, stream);
            for (const auto& part : parts) {
                const auto* bytes = static_cast<const uint8_t*>(part.p);
                if (part.n) fresh->key.insert(fresh->key.end(), bytes, bytes + part.n);
            }
            fresh->made.on(stream);
            kept.push_back(std::move(fresh));  // (nothing is kept of a call that fails before)
            tbp = kept.back().get();
        }
    }
    const GbTables& tb = *tbp;
    // A sparse tile keeps a hit's sum without its term, at most threshold - term; sums stay below
    // 2^15, so two bytes always hold one.  Where sum + term can pass the end of int32 any sum is kept.
    const bool wraps = sink && tb.most_term > INT32_MAX - kMaxHalf;
    const FastKernel kern = wraps  ? fast_kernel<true, true>(has_prior, wide)
                            : sink ? fast_kernel<true, false>(has_prior, wide)
                                   : fast_kernel<false, false>(has_prior, wide);
    const bool score16 = sink && (wraps || int64_t(sink->thresh) - tb.least_term > 255);

    const int tuned_choice =
        t_force_rc ? -1
                   : tuned_lookup(sink ? "sparse|" + gb_shape_key(qs, rs, has_prior)
                                       : gb_shape_key(qs, rs, has_prior));
    RefPlan* rpp = nullptr;
    FastSmem sm{};
    auto layout = [&](const RefPlan& rp) {
        return fast_smem(prof_bytes(qs.max_len, rp.max_spread, wide), int(rp.max_slab), rp.rc, W1,
                         rp.max_tasks, sink ? (score16 ? 2 : 1) : 0);
    };
    if (fast) {
        const int want_rc = t_force_rc ? t_force_rc : (tuned_choice >= 0 ? kRcCandidates[tuned_choice] : 0);
        // A resident set keeps a plan per width it is called with; the tuner's trials share one.
        RefPlans* own = rs.owns ? &plan_slot<RefPlans>(rs.gb_ref_plan, rs.gb_ref_plan, true) : nullptr;
        if (own)
            for (auto& p : own->of)
                if (!want_rc || p->rc == want_rc) rpp = p.get();
        std::unique_ptr<RefPlan> added;
        if (!rpp && own && !t_trial_rc) {
            added = std::make_unique<RefPlan>();
            rpp = added.get();
        }
        if (!rpp) rpp = &plan_slot<RefPlan>(own ? ctx.trial_ref_plan : ctx.tmp_ref_plan,
                                            own ? ctx.trial_ref_plan : ctx.tmp_ref_plan, false);
        RefPlan& rp = *rpp;
        if (rp.uid != rs.uid || (want_rc && rp.rc != want_rc)) {
            Phase ph("ref_plan");
            // Chunk width: the autotuner's measured choice when there is one; otherwise the
            // widest (best warp fill) that still reaches the highest CTA residency the
            // kernel's registers allow, checked with the occupancy calculator.
            int best_rc = 0, best_blocks = -1;
            std::vector<int> widths(kRcCandidates + 1, kRcCandidates + kNumRc);
            if (want_rc) widths.insert(widths.begin(), want_rc);
            for (int rc : widths) {
                build_ref_plan(rp, rs, rc);
                const int bytes = layout(rp).total;
                if (bytes > ctx.max_smem_optin) continue;
                if (rc == want_rc) {
                    best_rc = rc;
                    break;
                }
                int blocks = 0;
                ensure_smem_limit(reinterpret_cast<const void*>(kern), size_t(bytes));
                STB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kern, kThreads,
                                                                       size_t(bytes)));
                if (blocks > best_blocks) {
                    best_blocks = blocks;
                    best_rc = rc;
                }
                if (blocks >= kTargetBlocks[sink != nullptr]) break;
            }
            rp.uid = 0;  // stays so when no width fits shared memory: the general kernel runs
            if (best_rc) {
                if (rp.rc != best_rc) build_ref_plan(rp, rs, best_rc);
                std::vector<int4> up(rp.chunks);
                up.insert(up.end(), rp.tasks.begin(), rp.tasks.end());
                int4* d_plan = rp.d_plan.as<int4>(up.size(), stream);
                h2d(d_plan, up.data(), sizeof(int4) * up.size(), stream);
                uint32_t* meta = rp.d_meta.as<uint32_t>(size_t(K), stream);
                uint8_t* slab = rp.d_slab.as<uint8_t>(size_t(rp.slab_bytes) + 16, stream);
                const int4* tasks = d_plan + rp.nchunks;
                const bool few = rp.nchunks <= 4;  // beyond, a block per task fills more of the GPU
                (few ? chunk_order_kernel<true> : chunk_order_kernel<false>)<<<unsigned(rp.nchunks), 256, 0, stream>>>(
                    rs.d_len, K, rp.rc, rs.max_len, meta, rs.d_bytes, rs.d_off, d_plan, tasks, slab);
                STB_CUDA(cudaGetLastError());
                if (!few) {
                    ref_slab_kernel<<<unsigned(rp.ntasks), 128, 0, stream>>>(rs.d_bytes, rs.d_off, meta, tasks,
                                                                             rp.rc, slab);
                    STB_CUDA(cudaGetLastError());
                }
                note_launch(nullptr, few ? 1 : 2);
                if (added) rp.made.on(stream);
                rp.uid = rs.uid;
            }
        }
        sm = layout(rp);
        fast = rp.uid == rs.uid && sm.total <= ctx.max_smem_optin;
        if (added && fast) own->of.push_back(std::move(added));
    }

    if (!sink && !out_d) fail(ST_EINVAL, "seqtree_b200: null output buffer");
    if (!fast && sink && sink->ordered)
        fail(ST_ECUDA, "seqtree_b200: internal error: the ordered sparse form needs the fast kernel");
    if (!fast) {
        ScratchTurn turn(ctx, stream);
        int32_t* d_pen = ctx.table_buf.as<int32_t>(pen.size());
        h2d(d_pen, pen.data(), pen.size() * 4, stream);
        int32_t* d_prior = nullptr;
        if (has_prior) {
            d_prior = ctx.prior_buf.as<int32_t>(size_t(prior_len));
            h2d(d_prior, prior, size_t(prior_len) * 4, stream);
        }
        const int64_t rows = (r1 < 0 ? N : r1) - r0;
        GeneralArgs g{qs.d_bytes, qs.d_off, rs.d_bytes, rs.d_off, r0, rows, K, d_pen, A, go, ge,
                      d_prior, W1p, out_d, sink ? *sink : SparseSink{}};
        const int64_t blocks = std::min<int64_t>(ceil_div(rows * K, 256), int64_t(ctx.num_sms) * 16);
        if (sink)
            gapblock_general_kernel<true><<<unsigned(blocks), 256, size_t(A) * A * 4, stream>>>(g);
        else
            gapblock_general_kernel<false><<<unsigned(blocks), 256, size_t(A) * A * 4, stream>>>(g);
        STB_CUDA(cudaGetLastError());
        note_launch(sink ? "gapblock_general_kernel<sparse>" : "gapblock_general_kernel");
        return;
    }
    RefPlan& rp = *rpp;

    // Query pairs and their profile (rebuilt when the set or the penalty grid changes).
    const bool row_block = r0 != 0 || (r1 >= 0 && r1 != N);
    QueryPlan& qp = row_block ? plan_slot<QueryPlan>(ctx.tmp_block_plan, ctx.tmp_block_plan, false)
                              : plan_slot<QueryPlan>(qs.gb_query_plan, ctx.tmp_query_plan, qs.owns);
    if (qp.uid != qs.uid || qp.r0 != r0 || qp.r1 != (row_block ? r1 : -1)) {
        Phase ph("query_plan");
        build_query_plan(qp, qs, stream, r0, row_block ? r1 : -1);
    }
    const uint32_t* prof = nullptr;
    {
        std::vector<uint8_t> key(sizeof(int) * 2 + pen.size() * 4);
        const int hdr[2] = {A, int(wide)};
        std::memcpy(key.data(), hdr, sizeof hdr);
        std::memcpy(key.data() + sizeof hdr, pen.data(), pen.size() * 4);
        // a resident set keeps the profiles of its first grids; a transient set's and a row block's plan has one
        const bool kept = qs.owns && !row_block;
        Profile* found = nullptr;
        for (auto& p : qp.profiles)
            if (!kept || p->key == key) found = p.get();
        if (kept && (found ? found == qp.profiles.back().get() && qp.profiles.size() == kMaxProfiles
                           : qp.profiles.size() + 1 >= kMaxProfiles))
            refuse_capture(stream);
        if (!found || found->key != key) {
            const size_t words = size_t(qp.prof_rows) * kQuads * kRow * (wide ? 2 : 1);
            std::unique_ptr<Profile> added;
            if (!found && qp.profiles.size() < kMaxProfiles) {
                added = std::make_unique<Profile>();
                found = added.get();
            } else if (!found) {
                STB_CUDA(cudaDeviceSynchronize());  // any stream's kernels may read it
                found = qp.profiles.back().get();
            }
            found->key.clear();  // set again once the profile kernel is enqueued
            uint32_t* p = found->buf.as<uint32_t>(words, stream);
            qp.made.need(now);
            const int4* quads = static_cast<const int4*>(qp.d_plan.ptr);
            const int4* slices = quads + qp.quads.size();
            auto fill = wide ? profile_kernel<true> : profile_kernel<false>;
            fill<<<unsigned(qp.slices.size()), 256, 0, stream>>>(
                qs.d_bytes, qs.d_off, quads, slices, tb.pen, A,
                uint32_t(maxpen), p);
            STB_CUDA(cudaGetLastError());
            note_launch(nullptr);
            if (kept) found->made.on(stream);
            found->key = key;
            if (added) qp.profiles.push_back(std::move(added));
        }
        found->made.need(now);
        prof = static_cast<const uint32_t*>(found->buf.ptr);
    }
    rp.made.need(now);
    qp.made.need(now);

    auto* err = reinterpret_cast<unsigned long long*>(ctx.flags_d + 8);
    if (qs.owns || rs.owns) STB_CUDA(cudaMemsetAsync(err, 0, 8, stream));  // host calls cleared it

    FastArgs fa{};
    fa.prof = prof;
    fa.slab = static_cast<uint8_t*>(rp.d_slab.ptr);
    fa.rlen = rs.d_len;
    fa.K = K;
    fa.rc = rp.rc;
    fa.quads = static_cast<int4*>(qp.d_plan.ptr);
    fa.slices = fa.quads + qp.quads.size();
    fa.nslices = int64_t(qp.slices.size());
    fa.ref_meta = static_cast<uint32_t*>(rp.d_meta.ptr);
    fa.chunks = static_cast<int4*>(rp.d_plan.ptr);
    fa.tasks = fa.chunks + rp.nchunks;
    fa.sm = sm;
    fa.score16 = score16;
    fa.spread = rp.max_spread;
    fa.prior2 = has_prior ? tb.prior2 : nullptr;
    fa.ftab = tb.ftab;
    fa.W1 = W1;
    fa.pstride = prior_stride(W1);
    fa.out = out_d;
    fa.err = err;
    if (sink && sink->ordered) {
        const int64_t rows = (r1 < 0 ? N : r1) - r0;
        if (rows * int64_t(rp.nchunks) > sink->piece_cap)
            fail(ST_ECUDA, "seqtree_b200: internal error: sparse piece table too small");
        sink->nchunks = rp.nchunks;
        sink->row0 = r0;
    }
    if (sink) fa.sink = *sink;

    dim3 grid(unsigned(rp.nchunks), unsigned(fa.nslices));
    if (fa.nslices > 65535) {
        // slices split over y and z (the kernel skips the padding of the last z layer)
        grid.y = 65535;
        grid.z = unsigned(ceil_div(fa.nslices, 65535));
        if (grid.z > 65535) fail(ST_EINVAL, "seqtree_b200: too many queries for one launch");
    }
    ensure_smem_limit(reinterpret_cast<const void*>(kern), size_t(sm.total));
    kern<<<grid, kThreads, size_t(sm.total), stream>>>(fa);
    STB_CUDA(cudaGetLastError());
    note_launch(sink ? "gapblock_fast_kernel<sparse>" : "gapblock_fast_kernel");
    // The timeout flag is read by the caller after its synchronisation point.
}

}  // namespace

void gapblock_sets(st_seqset_s& qs, st_seqset_s& rs, const int32_t* penalty, int32_t matrix_size,
                   int32_t go, int32_t ge, const int32_t* prior, int64_t prior_len,
                   uint32_t prior_width, int32_t* out_d, cudaStream_t stream) {
    auto run = [&] {
        gapblock_run(qs, rs, penalty, matrix_size, go, ge, prior, prior_len, prior_width, out_d,
                     nullptr, stream);
    };
    // Only the fast kernel has a chunk width to choose (non-negative penalties, lengths <= 64;
    // the remaining range checks happen inside and fall back to the general kernel).
    bool nonneg = true;
    const int A = qs.alphabet >= 0 ? alphabet_size(qs.alphabet) : 0;
    if (penalty && matrix_size == A)
        for (int i = 0; i < A * A; ++i) nonneg &= penalty[i] >= 0;
    if (!nonneg || qs.count == 0 || rs.count == 0 || std::max(qs.max_len, rs.max_len) > 64 ||
        qs.alphabet < 0 || qs.alphabet != rs.alphabet || (penalty && matrix_size != A)) {
        run();
        return;
    }
    const bool has_prior = prior && prior_len > 0;
    const std::string key = gb_shape_key(qs, rs, has_prior);
    // Candidates: every chunk width.
    auto variant = [&](int c, int64_t rows, bool trial) {
        t_force_rc = c >= 0 ? kRcCandidates[c] : 0;  // -1: the static choice
        t_trial_rc = trial;
        try {
            if (rows < 0)
                run();
            else
                gapblock_run(qs, rs, penalty, matrix_size, go, ge, prior, prior_len, prior_width,
                             out_d, nullptr, stream, 0, rows);
        } catch (...) {
            t_force_rc = 0;
            t_trial_rc = false;
            throw;
        }
        t_force_rc = 0;
        t_trial_rc = false;
    };
    if (const int known = tuned_lookup(key); known >= 0) {
        variant(known, -1, false);
        return;
    }
    // A shape seen for the first time is tuned on its first query rows only (about
    // kTuneSlicePairs pairs, written into their own rows of the result), so the first call costs
    // the variants' runs on that slice rather than on the whole matrix; the chosen variant then
    // computes the whole matrix.
    const int64_t slice = std::min<int64_t>(
        qs.count, std::max<int64_t>(2 * kSliceQ, kTuneSlicePairs / std::max<int64_t>(rs.count, 1)));
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    STB_CUDA(cudaStreamIsCapturing(stream, &cs));
    const bool tunes = tuning_enabled() && cs == cudaStreamCaptureStatusNone;
    if (slice < qs.count && tunes) {
        const int c = tuned_run(key, kNumRc, -1, [&](int v) { variant(v, slice, true); }, stream);
        variant(c, -1, false);
        return;
    }
    tuned_run(key, kNumRc, -1, [&](int c) { variant(c, -1, tunes); }, stream);
}

// Scores of listed pairs (device index arrays) into out_d; the general int32 kernel's
// arithmetic, so any lengths and penalties.
void gapblock_pairs_sets(st_seqset_s& qs, st_seqset_s& rs, const int32_t* qi_d, const int32_t* ri_d,
                         int64_t n, const int32_t* penalty, int32_t matrix_size, int32_t go,
                         int32_t ge, const int32_t* prior, int64_t prior_len, uint32_t prior_width,
                         int32_t* out_d, int32_t* pos_d, cudaStream_t stream) {
    if (go < 0 || ge < 0) fail(ST_EINVAL, "gap_open and gap_extend must be >= 0");
    if (qs.alphabet < 0 || qs.alphabet != rs.alphabet)
        fail(ST_EINVAL, "seqtree_b200: gap-block sets must be encoded with one alphabet");
    const int A = alphabet_size(qs.alphabet);
    if (penalty && matrix_size != A) fail(ST_EINVAL, "matrix size does not match the alphabet");
    if (n < 0) fail(ST_EINVAL, "seqtree_b200: negative pair count");
    if (n == 0) return;
    const int64_t W1p = int64_t(prior_width) + 1;
    const bool has_prior = prior && prior_len > 0;
    if (has_prior) {
        if (prior_len != W1p * W1p * W1p)
            fail(ST_EINVAL, "prior table must have (prior_width + 1)^3 entries");
        if (uint32_t(std::max(qs.max_len, rs.max_len)) > prior_width)
            fail(ST_EINVAL, "a sequence is longer than the prior table's width");
    }
    Context& ctx = context();
    std::vector<int32_t> pen(size_t(A) * A);
    for (int x = 0; x < A; ++x)
        for (int y = 0; y < A; ++y) pen[size_t(x) * A + y] = penalty ? penalty[x * A + y] : int32_t(x != y);
    // Tables kept per device by content, so repeated calls upload nothing (and can be captured in a CUDA graph
    // once warmed up); prior cubes as the matrix tables: 16 are never rewritten, one more changes hands.
    struct PairPrior {
        std::vector<int32_t> cube;
        OwnedBuf buf;
        Made made;
    };
    constexpr size_t kMaxPriors = 17;
    static std::mutex mu;
    static auto& all = *new std::map<int, std::vector<std::unique_ptr<PairPrior>>>;  // (until the process exits)
    StreamScratch pen_mem;
    const int32_t* d_pen = kept_table(ctx, pen, stream, pen_mem);
    const int32_t* d_prior = nullptr;
    if (has_prior) {
        std::vector<std::unique_ptr<PairPrior>>* kept;
        {
            std::lock_guard<std::mutex> lk(mu);
            kept = &all[ctx.device];
        }
        auto it = std::find_if(kept->begin(), kept->end(), [&](const auto& p) {
            return int64_t(p->cube.size()) == prior_len &&
                   std::memcmp(p->cube.data(), prior, size_t(prior_len) * 4) == 0;
        });
        const bool found = it != kept->end();
        if (found ? it + 1 == kept->end() && kept->size() == kMaxPriors : kept->size() + 1 >= kMaxPriors)
            refuse_capture(stream);
        if (!found) {
            auto fresh = std::make_unique<PairPrior>();
            if (kept->size() == kMaxPriors) {
                STB_CUDA(cudaDeviceSynchronize());  // any stream's kernels may read it
                fresh = std::move(kept->back());
                kept->pop_back();
            }
            h2d(fresh->buf.as<int32_t>(size_t(prior_len), stream), prior, size_t(prior_len) * 4, stream);
            fresh->cube.assign(prior, prior + prior_len);
            fresh->made.on(stream);
            kept->push_back(std::move(fresh));
            it = kept->end() - 1;
        }
        (*it)->made.need(stream);
        d_prior = static_cast<const int32_t*>((*it)->buf.ptr);
    }
    const int64_t blocks = std::min<int64_t>(ceil_div(n, 256), int64_t(ctx.num_sms) * 16);
    gapblock_pairs_kernel<<<unsigned(blocks), 256, size_t(A) * A * 4, stream>>>(
        qs.d_bytes, qs.d_off, rs.d_bytes, rs.d_off, qi_d, ri_d, n, d_pen, A, go, ge, d_prior, W1p,
        out_d, pos_d);
    STB_CUDA(cudaGetLastError());
    note_launch("gapblock_pairs_kernel");
}

// ---------------------------------------------------------------------------- sparse --------
namespace {

int bits_for(int64_t n) {  // bits to hold 0..n-1 (at least 1)
    int b = 1;
    while (b < 62 && (int64_t(1) << b) < n) ++b;
    return b;
}

}  // namespace

// Hits of one query-row block: the kernel appends (key, score) pairs, a radix sort orders them by
// key (row-major), and csr_block_kernel writes the block's rows of indptr (offset by `base`) and ref ids.
// The block's ref ids and scores land at `base` in the result arrays.
namespace {

__global__ void csr_block_kernel(const unsigned long long* __restrict__ keys, int64_t H, int shift,
                                 int64_t row0, int64_t rows, int64_t base,
                                 int64_t* __restrict__ indptr, int32_t* __restrict__ ref_ids) {
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    const unsigned long long mask = (1ull << shift) - 1;
    for (int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; t <= rows || t < H;
         t += stride) {
        if (t <= rows) {
            const unsigned long long want = static_cast<unsigned long long>(row0 + t) << shift;
            int64_t lo = 0, hi = H;
            while (lo < hi) {
                const int64_t mid = (lo + hi) >> 1;
                if (keys[mid] < want) lo = mid + 1;
                else hi = mid;
            }
            indptr[row0 + t] = base + lo;
        }
        if (t < H) ref_ids[base + t] = int32_t(keys[t] & mask);
    }
}

// Ordered form, step 1: hits of each row of the block (the sum of its pieces), one warp per row.
__global__ void piece_rows_kernel(const int32_t* __restrict__ piece_cnt, int64_t rows, int nchunks,
                                  int64_t* __restrict__ rowcnt) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = (int64_t(gridDim.x) * blockDim.x) >> 5;
    for (int64_t r = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; r < rows; r += nw) {
        const int32_t* pc = piece_cnt + r * nchunks;
        long long sum = 0;
        for (int c = lane; c < nchunks; c += 32) sum += pc[c];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) rowcnt[r] = sum;
    }
}

// Ordered form, step 2: the block's CSR rows.  start[r] is the exclusive prefix of the rows' hits
// inside the block (start[rows] the block's total) and base the hits of earlier blocks.  A warp
// walks its row's pieces in chunk order -- ascending columns -- and copies each (ref id, score)
// run into place.
__global__ void piece_copy_kernel(const int2* __restrict__ seg, const int64_t* __restrict__ piece_off,
                                  const int32_t* __restrict__ piece_cnt,
                                  const int64_t* __restrict__ start, int64_t rows, int nchunks,
                                  int64_t row0, int64_t base, int64_t* __restrict__ indptr,
                                  int32_t* __restrict__ ref_ids, int32_t* __restrict__ scores) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int64_t nw = (int64_t(gridDim.x) * blockDim.x) >> 5;
    for (int64_t r = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; r < rows; r += nw) {
        long long pos = base + start[r];
        if (lane == 0) {
            indptr[row0 + r] = pos;
            if (r == rows - 1) indptr[row0 + rows] = base + start[rows];
        }
        for (int c0 = 0; c0 < nchunks; c0 += 32) {
            const int c = c0 + lane;
            const int32_t cnt = c < nchunks ? piece_cnt[r * nchunks + c] : 0;
            const long long src = cnt > 0 ? piece_off[r * nchunks + c] : 0;
            long long incl = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const long long t = __shfl_up_sync(full, incl, o);
                if (lane >= o) incl += t;
            }
            const long long dst = pos + incl - cnt;
            uint32_t m = __ballot_sync(full, cnt > 0);
            while (m) {
                const int L = __ffs(int(m)) - 1;
                m &= m - 1;
                const int32_t n = __shfl_sync(full, cnt, L);
                const long long s0 = __shfl_sync(full, src, L);
                const long long d0 = __shfl_sync(full, dst, L);
                for (int i = lane; i < n; i += 32) {
                    const int2 h = seg[s0 + i];
                    ref_ids[d0 + i] = h.x;
                    scores[d0 + i] = h.y;
                }
            }
            pos += __shfl_sync(full, incl, 31);
        }
    }
}

// Hits one sort takes at most (2^28, about 10 GB of scratch); larger outputs are produced in
// query-row blocks.  SEQTREE_B200_SPARSE_BLOCK_HITS lowers it (at least 1024), e.g. to bound the
// scratch memory.
uint64_t max_block_hits() {
    uint64_t v = uint64_t(1) << 28;
    if (const char* e = std::getenv("SEQTREE_B200_SPARSE_BLOCK_HITS")) {
        const long long x = std::atoll(e);
        if (x > 0) v = std::min<uint64_t>(v, std::max<uint64_t>(uint64_t(x), 1024));
    }
    return v;
}

// Hits one block of the ordered form holds (2^31: 16 GB of segments), or the same override as
// the sort's cap, so that the row-block path can be exercised on small inputs.
uint64_t max_segment_hits() {
    const char* e = std::getenv("SEQTREE_B200_SPARSE_BLOCK_HITS");
    return (e && std::atoll(e) > 0) ? max_block_hits() : (uint64_t(1) << 31);
}

}  // namespace

void gapblock_sparse_sets(st_seqset_s& qs, st_seqset_s& rs, const int32_t* penalty,
                          int32_t matrix_size, int32_t go, int32_t ge, const int32_t* prior,
                          int64_t prior_len, uint32_t prior_width, int32_t max_penalty,
                          st_hits_s& hits, cudaStream_t stream) {
    if (max_penalty < 0) fail(ST_EINVAL, "max_penalty must be >= 0");
    Context& ctx = context();
    const int64_t N = qs.count, K = rs.count;
    hits.rows = N;
    hits.cols = K;
    hits.nnz = 0;
    int64_t* indptr = hits.indptr.as<int64_t>(size_t(N) + 1);
    if (N == 0 || K == 0) {
        // the dense call's checks still apply (they come before its empty-shape return)
        gapblock_run(qs, rs, penalty, matrix_size, go, ge, prior, prior_len, prior_width, nullptr,
                     nullptr, stream);
        STB_CUDA(cudaMemsetAsync(indptr, 0, sizeof(int64_t) * size_t(N + 1), stream));
        return;
    }
    ScratchTurn turn(ctx, stream);
    const int shift = bits_for(K);
    if (shift + bits_for(N) > 63) fail(ST_EINVAL, "seqtree_b200: matrix too large for sparse keys");
    const int end_bit = shift + bits_for(N);
    const uint64_t kMaxBlockHits = max_block_hits();
    auto* count = reinterpret_cast<unsigned long long*>(ctx.flags_d + 10);
    const bool ordered = fast_form_possible(qs, rs, penalty, matrix_size);

    // The fast kernel's chunk width and launch form are tuned once per shape, as for the dense
    // matrix, but on a slice of about 2e9 pairs of rows: every variant counts the slice's hits
    // into the sink (what it stores is overwritten by the passes below).
    {
        const bool has_prior = prior && prior_len > 0;
        const std::string skey = "sparse|" + gb_shape_key(qs, rs, has_prior);
        bool nonneg = qs.alphabet >= 0 && qs.alphabet == rs.alphabet &&
                      std::max(qs.max_len, rs.max_len) <= 64;
        const int A = nonneg ? alphabet_size(qs.alphabet) : 0;
        if (penalty && matrix_size != A) nonneg = false;
        if (nonneg && penalty)
            for (int i = 0; i < A * A; ++i) nonneg &= penalty[i] >= 0;
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        STB_CUDA(cudaStreamIsCapturing(stream, &cs));
        if (nonneg && tuning_enabled() && cs == cudaStreamCaptureStatusNone && tuned_lookup(skey) < 0) {
            const int64_t tr1 = std::min<int64_t>(N, std::max<int64_t>(64, int64_t(2000000000) / K));
            const uint64_t tcap = std::min<uint64_t>(std::max<uint64_t>(hits.cap_hint, uint64_t(1) << 20),
                                                     kMaxBlockHits);
            SparseSink ts{};
            ts.count = count;
            ts.cap = tcap;
            ts.shift = shift;
            ts.thresh = max_penalty;
            if (ordered) {
                // room for hits at up to 1/8 density, so that the variants are timed with their
                // hit writes (a tile whose hits do not fit only counts them)
                ts.cap = std::min<uint64_t>(max_segment_hits(),
                                            std::max<uint64_t>(tcap, uint64_t(tr1) * uint64_t(K) / 8));
                ts.ordered = 1;
                ts.seg = ctx.sp_keys.as<int2>(size_t(ts.cap));
                ts.piece_cap = (tr1 == N ? N : tr1) * ceil_div(K, kRcCandidates[kNumRc - 1]);
                ts.piece_off = ctx.sp_sorted.as<int64_t>(size_t(ts.piece_cap));
                ts.piece_cnt = ctx.sp_vals.as<int32_t>(size_t(ts.piece_cap));
            } else {
                ts.keys = ctx.sp_keys.as<unsigned long long>(size_t(tcap));
                ts.vals = ctx.sp_vals.as<int32_t>(size_t(tcap));
            }
            tuned_run(skey, kNumRc, -1, [&](int c) {
                t_force_rc = c >= 0 ? kRcCandidates[c] : 0;
                t_trial_rc = true;
                try {
                    STB_CUDA(cudaMemsetAsync(count, 0, sizeof(unsigned long long), stream));
                    gapblock_run(qs, rs, penalty, matrix_size, go, ge, prior, prior_len,
                                 prior_width, nullptr, &ts, stream, 0, tr1 == N ? -1 : tr1);
                } catch (...) {
                    t_force_rc = 0;
                    t_trial_rc = false;
                    throw;
                }
                t_force_rc = 0;
                t_trial_rc = false;
            }, stream);
        }
    }

    if (ordered) {
        // Ordered form: no sort.  One block of all rows in the usual case; blocks of rows when
        // the segments (max_segment_hits) or the piece table (2^28 entries) would not hold them.
        const uint64_t seg_cap_max = max_segment_hits();
        const int64_t most_chunks = ceil_div(K, kRcCandidates[kNumRc - 1]);
        const int64_t piece_rows = std::max<int64_t>(1, (int64_t(1) << 28) / most_chunks);
        int64_t r0 = 0, rows = std::min<int64_t>(
            hits.block_rows_hint > 0 ? hits.block_rows_hint : N, piece_rows);
        int64_t first_rows = 0, nblocks = 0, total = 0;
        uint64_t cap = std::min<uint64_t>(std::max<uint64_t>(hits.cap_hint, uint64_t(1) << 20),
                                          seg_cap_max);
        bool exact_retry = false;
        while (r0 < N) {
            const int64_t r1 = std::min<int64_t>(N, r0 + rows);
            SparseSink sink{};
            sink.ordered = 1;
            sink.count = count;
            sink.cap = cap;
            sink.shift = shift;
            sink.thresh = max_penalty;
            sink.seg = ctx.sp_keys.as<int2>(size_t(cap));
            sink.piece_cap = (r1 - r0) * most_chunks;
            sink.piece_off = ctx.sp_sorted.as<int64_t>(size_t(sink.piece_cap));
            sink.piece_cnt = ctx.sp_vals.as<int32_t>(size_t(sink.piece_cap));
            STB_CUDA(cudaMemsetAsync(ctx.flags_d + 8, 0, 8 * sizeof(int64_t), stream));
            gapblock_run(qs, rs, penalty, matrix_size, go, ge, prior, prior_len, prior_width,
                         nullptr, &sink, stream, r0, r1 == N && r0 == 0 ? -1 : r1);
            STB_CUDA(cudaMemcpyAsync(ctx.flags_h + 8, ctx.flags_d + 8, 8 * sizeof(int64_t),
                                     cudaMemcpyDeviceToHost, stream));
            STB_CUDA(cudaStreamSynchronize(stream));
            if (ctx.flags_h[8] != 0)
                fail(ST_ETIMEOUT,
                     "seqtree_b200: a bounded device-side wait gave up (shared-memory staging)");
            const uint64_t H = static_cast<uint64_t>(ctx.flags_h[10]);
            if (H > cap) {
                if (exact_retry) fail(ST_ECUDA, "seqtree_b200: sparse hit count changed between passes");
                const int64_t nrows = r1 - r0;
                if (H <= seg_cap_max || nrows == 1) {
                    cap = H;  // the same block at its exact size (one row holds < 2^31 hits)
                    exact_retry = true;
                } else {
                    const double per_row = double(H) / double(nrows);
                    rows = std::max<int64_t>(
                        1, std::min<int64_t>(nrows - 1, int64_t(0.75 * double(seg_cap_max) / per_row)));
                }
                continue;
            }
            exact_retry = false;
            const int64_t nrows = r1 - r0;
            const size_t need = size_t(total + int64_t(H) + 1);
            hits.ref_ids.grow_keep(need * sizeof(int32_t), size_t(total) * sizeof(int32_t), stream);
            hits.scores.grow_keep(need * sizeof(int32_t), size_t(total) * sizeof(int32_t), stream);
            int64_t* rowcnt = ctx.work_b.as<int64_t>(size_t(2 * (nrows + 1)));
            int64_t* start = rowcnt + (nrows + 1);
            const unsigned wblocks =
                unsigned(std::min<int64_t>(ceil_div(nrows * 32, 256), int64_t(ctx.num_sms) * 16));
            STB_CUDA(cudaMemsetAsync(rowcnt + nrows, 0, sizeof(int64_t), stream));
            piece_rows_kernel<<<wblocks, 256, 0, stream>>>(sink.piece_cnt, nrows, sink.nchunks,
                                                           rowcnt);
            STB_CUDA(cudaGetLastError());
            size_t temp = 0;
            STB_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, temp, rowcnt, start, int(nrows + 1),
                                                   stream));
            void* d_temp = ctx.sp_temp.as<uint8_t>(temp + 16);
            STB_CUDA(cub::DeviceScan::ExclusiveSum(d_temp, temp, rowcnt, start, int(nrows + 1),
                                                   stream));
            piece_copy_kernel<<<wblocks, 256, 0, stream>>>(
                sink.seg, sink.piece_off, sink.piece_cnt, start, nrows, sink.nchunks, r0, total,
                indptr, static_cast<int32_t*>(hits.ref_ids.ptr),
                static_cast<int32_t*>(hits.scores.ptr));
            STB_CUDA(cudaGetLastError());
            note_launch(nullptr, 2);
            total += int64_t(H);
            if (nblocks++ == 0) first_rows = nrows;
            const double per_row = double(std::max<uint64_t>(H, 1)) / double(nrows);
            rows = std::min<int64_t>(piece_rows,
                                     std::max<int64_t>(1, int64_t(0.75 * double(seg_cap_max) / per_row)));
            cap = std::min<uint64_t>(
                std::max<uint64_t>(cap, uint64_t(per_row * double(rows) * 1.25) + 1024), seg_cap_max);
            r0 = r1;
        }
        hits.nnz = total;
        hits.block_rows_hint = nblocks > 1 ? first_rows : 0;
        hits.cap_hint = std::max<uint64_t>(
            hits.cap_hint, std::min<uint64_t>(uint64_t(total) + uint64_t(total) / 8, seg_cap_max));
        return;
    }

    // One block of all rows when the hits fit one sort (the usual case: the set's cached plans
    // are used and nothing is copied); otherwise blocks sized from the hit density seen so far.
    int64_t r0 = 0, rows = hits.block_rows_hint > 0 ? hits.block_rows_hint : N;
    int64_t first_rows = 0, nblocks = 0;
    uint64_t cap = std::min<uint64_t>(std::max<uint64_t>(hits.cap_hint, uint64_t(1) << 20),
                                      kMaxBlockHits);
    int64_t total = 0;
    bool exact_retry = false;
    while (r0 < N) {
        const int64_t r1 = std::min<int64_t>(N, r0 + rows);
        SparseSink sink{};
        sink.keys = ctx.sp_keys.as<unsigned long long>(size_t(cap));
        sink.vals = ctx.sp_vals.as<int32_t>(size_t(cap));
        sink.count = count;
        sink.cap = cap;
        sink.shift = shift;
        sink.thresh = max_penalty;
        STB_CUDA(cudaMemsetAsync(ctx.flags_d + 8, 0, 8 * sizeof(int64_t), stream));
        gapblock_run(qs, rs, penalty, matrix_size, go, ge, prior, prior_len, prior_width, nullptr,
                     &sink, stream, r0, r1 == N && r0 == 0 ? -1 : r1);
        STB_CUDA(cudaMemcpyAsync(ctx.flags_h + 8, ctx.flags_d + 8, 8 * sizeof(int64_t),
                                 cudaMemcpyDeviceToHost, stream));
        STB_CUDA(cudaStreamSynchronize(stream));
        if (ctx.flags_h[8] != 0)
            fail(ST_ETIMEOUT, "seqtree_b200: a bounded device-side wait gave up (shared-memory staging)");
        const uint64_t H = static_cast<uint64_t>(ctx.flags_h[10]);
        if (H > cap) {
            if (exact_retry) fail(ST_ECUDA, "seqtree_b200: sparse hit count changed between passes");
            const int64_t nrows = r1 - r0;
            if (H <= kMaxBlockHits || nrows == 1) {
                // same block at its exact size (a single row may exceed the block cap: its hits
                // are at most K < 2^31, what one sort takes)
                cap = H <= kMaxBlockHits ? std::min<uint64_t>(H + H / 8, kMaxBlockHits) : H;
                exact_retry = true;
            } else {  // fewer rows, sized to about 3/4 of a full sort
                const double per_row = double(H) / double(nrows);
                rows = std::max<int64_t>(
                    1, std::min<int64_t>(nrows - 1, int64_t(0.75 * double(kMaxBlockHits) / per_row)));
                cap = kMaxBlockHits;
            }
            continue;
        }
        exact_retry = false;
        // room for this block's results after the previous blocks'
        const size_t need = size_t(total + int64_t(H) + 1);
        hits.ref_ids.grow_keep(need * sizeof(int32_t), size_t(total) * sizeof(int32_t), stream);
        hits.scores.grow_keep(need * sizeof(int32_t), size_t(total) * sizeof(int32_t), stream);
        auto* ref_ids = static_cast<int32_t*>(hits.ref_ids.ptr);
        auto* scores = static_cast<int32_t*>(hits.scores.ptr);
        auto* sorted = ctx.sp_sorted.as<unsigned long long>(size_t(std::max<uint64_t>(H, 1)));
        if (H > 0) {
            size_t temp = 0;
            STB_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, temp, sink.keys, sorted, sink.vals,
                                                     scores + total, int(H), 0, end_bit, stream));
            void* d_temp = ctx.sp_temp.as<uint8_t>(temp + 16);
            STB_CUDA(cub::DeviceRadixSort::SortPairs(d_temp, temp, sink.keys, sorted, sink.vals,
                                                     scores + total, int(H), 0, end_bit, stream));
        }
        const int64_t work = std::max<int64_t>(r1 - r0 + 1, int64_t(H));
        const unsigned blocks =
            unsigned(std::min<int64_t>(ceil_div(work, 256), int64_t(ctx.num_sms) * 8));
        csr_block_kernel<<<blocks, 256, 0, stream>>>(sorted, int64_t(H), shift, r0, r1 - r0, total,
                                                     indptr, ref_ids);
        STB_CUDA(cudaGetLastError());
        note_launch(nullptr);
        total += int64_t(H);
        if (nblocks++ == 0) first_rows = r1 - r0;
        // next block: as many rows as this block's density says fit 3/4 of a sort
        const double per_row = double(std::max<uint64_t>(H, 1)) / double(r1 - r0);
        rows = std::max<int64_t>(1, int64_t(0.75 * double(kMaxBlockHits) / per_row));
        cap = std::min<uint64_t>(std::max<uint64_t>(cap, uint64_t(per_row * double(rows) * 1.25) + 1024),
                                 kMaxBlockHits);
        r0 = r1;
    }
    hits.nnz = total;
    hits.block_rows_hint = nblocks > 1 ? first_rows : 0;
    hits.cap_hint = std::max<uint64_t>(hits.cap_hint, std::min<uint64_t>(uint64_t(total) + uint64_t(total) / 8, kMaxBlockHits));
}

}  // namespace stb
