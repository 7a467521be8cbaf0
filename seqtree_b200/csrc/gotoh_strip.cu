// Gotoh alignment in row strips, one lane per reference (NW / SW with gap_extend <= gap_open).
//
// A warp scores two queries (neighbours in length order, packed int16x2) against 32 refs
// (neighbours in length order), one ref per lane.  The query's rows are cut into strips of R rows
// (R <= 48, even up to 24 and a multiple of 4 beyond, so fewer than 4 rows a strip are padding: 49 rows are two
// strips of 28); a lane keeps H and Y of the strip's rows in registers and walks the columns of its ref, so there are no
// shuffles, no ramp and no idle lanes, which is where the query-pair wavefront (pairwise.cu) loses
// its time: 31 of n + 31 steps, up to 31 padded rows and the per-step exchange.  Between strips the
// bottom row's (H, next X) pair of each column goes through a per-warp slice of global scratch
// (8 B per column and lane, read two columns ahead; 16 B of L2 traffic per R cell pairs).
//
// The bound is the ALU pipe (64 lanes/clk/SM, DPX included).  Per cell pair, with every state of
// (i, j) raised by (i + j) * extend in global mode and by j * extend in local mode:
//   MY = max(diag + s, Y)               1 DPX   (s carries the raise)
//   H  = max(MY, X [, floor])           1 DPX   (local: the raised zero of this column)
//   X' = max(MY + e - o, X)             1 DPX   global;  local: max(X - e, MY - o), the MY - o an
//                                               IMAD on the otherwise idle FMA pipe
//   Y' = max(H + e - o, Y)              1 DPX
// X' takes MY where the recurrence takes H = max(MY, X): X + e - o <= X (and X - o <= X - e), and a
// local floor of 0 can only start a gap below 0, which no later maximum takes.  This leaves one DPX
// per row on the dependent chain (X -> X'), so two or three warps per scheduler fill the pipe.
// One LDS per cell pair fetches the scores of both queries: the profile is [row][25 codes], so the
// lanes' codes fall into distinct banks, at an immediate offset from one register per column.
//
// Padding never needs a test in the loop.  Rows past a query and columns past a ref score 0 (plus
// the raise).  They lie after every real cell, so a global score read at (m, n) does not see them;
// in local mode a padded cell never exceeds the best cell before it.
//
// Measured, B200 at 1965 MHz, whole calls: 4,096 x 4,096 proteins (median 180 residues) global
// distance 128 -> 96 ms (query-pair wavefront -> this), local scores of 1,501 x 4,003 of them
// 66.7 -> 39.9 ms, 4,096 x 4,096 junctions (10-20) global distance 7.98 -> 0.71 ms (one int32
// thread per pair -> this).  ncu counts 4.26 ALU instructions per cell pair in global mode (4.7
// local; 4.75 on junctions, at 82 % ALU pipe activity).
#include <algorithm>
#include <climits>
#include <map>
#include <numeric>

#include "common.cuh"

namespace stb {

namespace {

constexpr int kStripWarps = 4;
constexpr int kProfW = 25;        // words per profile row: 24 codes and the padding code
constexpr int kPadCode = 24;
constexpr int kBias = 16384;      // local mode keeps both halves non-negative (IMAD adds both)

struct StripArgs {
    const uint8_t* qc;
    const int64_t* qoff;
    const int2* qpairs;       // longest first; x == y for a single
    int64_t nqp;
    const uint32_t* slab;     // per group of 32 refs: ceil(longest / 4) x 32 words, 4 codes * 4 each
    const int2* groups;       // per group: slab offset (in 32-word rows), its longest ref | 1 << 16
                              // when it has 32 refs of that length
    const int2* rmeta;        // refs (index, length), longest first
    int64_t K;
    int ngroups;
    int gpw;                  // groups a warp takes per unit
    int nchunks;              // units per query pair
    const int32_t* sim;       // A x A: s(a, b) + raise
    int A;
    int add;                  // score of a padded cell (the raise alone)
    int go, ge;
    uint32_t one;             // 1, opaque to the compiler: keeps x * one + c an IMAD
    int dist;
    const int64_t* q_self;
    const int64_t* r_self;
    int32_t* out;
    unsigned int* overflow;
    uint2* scratch;           // per warp of the grid: cols x 32 (H, X') pairs
    int64_t scratch_cols;
    unsigned long long* queue;  // zeroed; null when every CTA has one unit
};

__device__ __forceinline__ uint32_t dup16(int v) { return uint32_t(uint16_t(int16_t(v))) * 0x10001u; }

// Strips of at most `most` rows for m rows: how many, and rows per strip (even up to 24, then a
// multiple of 4).
__host__ __device__ inline void strip_shape(int m, int most, int& strips, int& rows) {
    strips = (m + most - 1) / most;
    if (strips < 1) strips = 1;
    rows = (m + strips - 1) / strips;
    rows = rows <= 24 ? (rows + 1) / 2 * 2 : (rows + 3) / 4 * 4;
    if (rows < 4) rows = 4;
}

// All groups of this warp's share of a unit: query pair (q.x, q.y) against refs of groups
// g0, g0 + kStripWarps, ... < g1.
template <int R, bool LOCAL>
__device__ __forceinline__ void strip_unit(const StripArgs& a, const uint32_t* s_prof, int strips, int2 qp,
                                           int m1, int m2, int g0, int g1, uint2* scr) {
    const int lane = threadIdx.x & 31;
    const uint32_t eo2 = dup16(a.ge - a.go), mge2 = dup16(-a.ge);
    const uint32_t mgo_add = 0u - uint32_t(a.go) * 0x10001u;  // subtracts go from both halves
    const uint32_t e2 = uint32_t(a.ge) * 0x10001u;
    auto ref_of = [&](int g) {
        const int64_t t = int64_t(g) * 32 + lane;
        return t < a.K ? a.rmeta[t] : make_int2(-1, 0);
    };
    if (g0 >= g1) return;
    int2 grp = a.groups[g0], ref = ref_of(g0);
    uint32_t head = a.slab[int64_t(grp.x) * 32 + lane];
    for (int g = g0; g < g1; g += kStripWarps) {
        const uint32_t* codes = a.slab + int64_t(grp.x) * 32 + lane;
        const int k = ref.x, n = ref.y, cols = grp.y & 0xFFFF;
        const bool one_length = (grp.y >> 16) != 0;
        const uint32_t first_codes = head;
        // the next group's head is on its way while this one runs
        if (g + kStripWarps < g1) {
            grp = a.groups[g + kStripWarps];
            ref = ref_of(g + kStripWarps);
            head = a.slab[int64_t(grp.x) * 32 + lane];
        }
        uint32_t c1 = 0u, c2 = 0u, best = 0u;
        for (int s = 0; s < strips; ++s) {
            const uint8_t* prof = reinterpret_cast<const uint8_t*>(s_prof + s * R * kProfW);
            const bool first = s == 0, last = s == strips - 1;
            uint32_t H[R], Y[R];
            const uint32_t h0 = LOCAL ? dup16(kBias) : eo2;
            const uint32_t y0 = LOCAL ? dup16(kBias + a.ge - a.go) : dup16(2 * (a.ge - a.go));
#pragma unroll
            for (int r = 0; r < R; ++r) {
                H[r] = h0;
                Y[r] = y0;
            }
            uint32_t diag = LOCAL ? h0 : (first ? 0u : eo2);
            // Top boundary of strip 0: H(0, j) and X(1, j).  Later strips read the scratch.
            uint32_t floor2 = dup16(kBias);  // local: the raised zero of column j
            uint2 top = make_uint2(eo2, y0);
            uint2 nxt = make_uint2(0u, 0u), nx2 = make_uint2(0u, 0u);
            if (!first) {
                nxt = scr[lane];
                if (cols > 1) nx2 = scr[32 + lane];
            }
            // rows of the two queries' last residues in this strip, or -1
            const int cr1 = (!LOCAL && (m1 - 1) / R == s) ? (m1 - 1) - s * R : -1;
            const int cr2 = (!LOCAL && (m2 - 1) / R == s) ? (m2 - 1) - s * R : -1;
            const bool capture = !LOCAL && (cr1 >= 0 || cr2 >= 0), mixed = capture && !one_length;
            uint32_t w = 0u, wn = first_codes;
            uint32_t nfl = 0u;  // local: -(j * extend) in both halves
            int je = 0;
            auto keep = [&] {  // the scores' halves, once column n is done
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    if (r == cr1) c1 = H[r];
                    if (r == cr2) c2 = H[r];
                }
            };
            auto column = [&](int j) {
                const uint8_t* pc = prof + (w & 0xFFu);
                w >>= 8;
                if constexpr (LOCAL) {
                    floor2 += e2;
                    je += a.ge;
                    nfl = dup16(-je);
                }
                if (!first) {
                    top = nxt;
                    nxt = nx2;
                    if (j + 2 < cols) nx2 = scr[(j + 2) * 32 + lane];
                } else if constexpr (LOCAL) {
                    top.x = floor2;
                    top.y = floor2 + mgo_add;
                }
                uint32_t x = top.y;
                uint32_t my = __viaddmax_s16x2(diag, *reinterpret_cast<const uint32_t*>(pc), Y[0]);
                uint32_t colmax = floor2, hprev = 0u;
                diag = top.x;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    uint32_t myn = 0u;
                    if (r + 1 < R)
                        myn = __viaddmax_s16x2(
                            H[r], *reinterpret_cast<const uint32_t*>(pc + (r + 1) * kProfW * 4),
                            Y[r + 1]);
                    uint32_t h;
                    if constexpr (LOCAL) {
                        h = __vimax3_s16x2(my, x, floor2);
                        x = __viaddmax_s16x2(x, mge2, my * a.one + mgo_add);
                        if (r & 1) colmax = __vimax3_s16x2(colmax, hprev, h);
                        hprev = h;
                    } else {
                        h = __vmaxs2(my, x);
                        x = __viaddmax_s16x2(my, eo2, x);
                    }
                    Y[r] = __viaddmax_s16x2(h, eo2, Y[r]);
                    H[r] = h;
                    my = myn;
                }
                if constexpr (LOCAL) best = __viaddmax_s16x2(colmax, nfl, best);
                if (!last) scr[j * 32 + lane] = make_uint2(H[R - 1], x);
                if (mixed && j + 1 == n) keep();
            };
            // Four columns per code word, not unrolled: a column is long enough to hide its loop, and
            // with a body per strip height the instruction cache holds single columns at best
            // (two at a time 0.71 against 0.69 ms on 4,096 x 4,096 junctions, four 0.74).
            int j = 0;
#pragma unroll 1
            for (; j + 4 <= cols; j += 4) {
                w = wn;
                if (j + 4 < cols) wn = codes[j * 8 + 32];
#pragma unroll 1
                for (int u = 0; u < 4; ++u) column(j + u);
            }
            w = wn;
#pragma unroll 1
            for (; j < cols; ++j) column(j);
            if (capture && !mixed) keep();
        }
        int v1, v2;
        if constexpr (LOCAL) {
            v1 = int(best & 0xFFFFu) - kBias;
            v2 = int(best >> 16) - kBias;
        } else {
            v1 = int(int16_t(uint16_t(c1 & 0xFFFFu))) - (m1 + n) * a.ge;
            v2 = int(int16_t(uint16_t(c2 >> 16))) - (m2 + n) * a.ge;
        }
        if (k >= 0) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (h == 1 && qp.y == qp.x) break;
                const int qi = h ? qp.y : qp.x;
                const int64_t sv = h ? v2 : v1;
                const int64_t v = a.dist ? a.q_self[qi] + a.r_self[k] - 2 * sv : sv;
                if (v < INT32_MIN || v > INT32_MAX)
                    atomicOr(a.overflow, 1u);
                else
                    a.out[int64_t(qi) * a.K + k] = int32_t(v);
            }
        }
    }
}

// Persistent CTAs take units (query pair, chunk of ref groups), longest pairs and refs first, from
// a counter (dealing them round-robin left CTAs with nothing but long refs: 120 against 97 ms on the
// proteins).  MAXR 48 is for queries longer than 32: three CTAs of four warps per SM by registers,
// and no spills in global mode.  Taller strips spill (64 rows: 160 ms) or, with the registers to
// hold them, leave two CTAs per SM (150 ms); 32 rows read and write the scratch more often (126 ms,
// all before the queue; 95.0 against 96.8 ms for 56 rows with it, local mode 116.8 against 114.0).
// MAXR 32 runs four CTAs and serves sets whose queries have at most 32 residues.

template <int MAXR, bool LOCAL>
__global__ void __launch_bounds__(kStripWarps * 32, MAXR == 48 ? 3 : 4)
gotoh_strip_kernel(const StripArgs a) {
    extern __shared__ uint32_t s_prof[];
    const int warp = threadIdx.x >> 5;
    uint2* scr = a.scratch + (int64_t(blockIdx.x) * kStripWarps + warp) * a.scratch_cols * 32;
    const int64_t units = a.nqp * a.nchunks;
    __shared__ unsigned long long s_next;
    for (int64_t u = blockIdx.x; u < units;) {
        const int64_t p = u / a.nchunks;
        const int chunk = int(u - p * a.nchunks);
        const int2 qp = a.qpairs[p];
        const int64_t o1 = a.qoff[qp.x], o2 = a.qoff[qp.y];
        const int m1 = int(a.qoff[qp.x + 1] - o1), m2 = int(a.qoff[qp.y + 1] - o2);
        int strips, R;
        strip_shape(max(m1, m2), MAXR, strips, R);
        __syncthreads();  // every warp is done with the previous unit's profile
        // the unit after this one is asked for now, so the answer is there when it is needed
        if (threadIdx.x == 0)
            s_next = a.queue ? gridDim.x + atomicAdd(a.queue, 1ull) : (unsigned long long)(units);
        for (int i = threadIdx.x; i < strips * R * kProfW; i += kStripWarps * 32) {
            const int row = i / kProfW, c = i - row * kProfW;
            int v1 = a.add, v2 = a.add;
            if (c < a.A) {
                if (row < m1) v1 = a.sim[int(a.qc[o1 + row]) * a.A + c];
                if (row < m2) v2 = a.sim[int(a.qc[o2 + row]) * a.A + c];
            }
            s_prof[i] = uint32_t(uint16_t(int16_t(v1))) | (uint32_t(uint16_t(int16_t(v2))) << 16);
        }
        __syncthreads();
        u = int64_t(s_next);
        const int span = kStripWarps * a.gpw;
        const int g0 = chunk * span + warp, g1 = min(a.ngroups, (chunk + 1) * span);
#define STB_STRIP(RR)                                                                          \
    case RR:                                                                                   \
        strip_unit<RR, LOCAL>(a, s_prof, strips, qp, m1, m2, g0, g1, scr);                     \
        break;
        switch (R) {
            STB_STRIP(4) STB_STRIP(6) STB_STRIP(8) STB_STRIP(10) STB_STRIP(12) STB_STRIP(14)
            STB_STRIP(16) STB_STRIP(18) STB_STRIP(20) STB_STRIP(22) STB_STRIP(24) STB_STRIP(28)
            STB_STRIP(32)
        }
        if constexpr (MAXR == 48)
            switch (R) { STB_STRIP(36) STB_STRIP(40) STB_STRIP(44) STB_STRIP(48) }
#undef STB_STRIP
    }
}

// Ref codes of every group: word [g][j / 4][lane] holds four columns' 4 * code (the padding code
// past a ref's end and past the last ref).
__global__ void strip_slab_kernel(const uint8_t* __restrict__ codes, const int64_t* __restrict__ off,
                                  const int2* __restrict__ meta, int64_t K,
                                  const int2* __restrict__ groups, uint32_t* __restrict__ slab) {
    const int g = blockIdx.x;
    const int2 grp = groups[g];
    for (int i = threadIdx.x; i < ((grp.y & 0xFFFF) + 3) / 4 * 32; i += blockDim.x) {
        const int lane = i & 31, j = (i >> 5) * 4;
        const int64_t t = int64_t(g) * 32 + lane;
        uint32_t w = 0u;
        const int2 ref = t < K ? meta[t] : make_int2(0, 0);
        const int k = ref.x, n = ref.y;
        for (int b = 0; b < 4; ++b) {
            const uint32_t c = j + b < n ? uint32_t(codes[off[k] + j + b]) : uint32_t(kPadCode);
            w |= (c * 4u) << (8 * b);
        }
        slab[int64_t(grp.x) * 32 + i] = w;
    }
}

// Launch plans of a set (they depend on its lengths and codes): the query side's pairs, longest
// first, and the ref side's order, groups and code slab.
struct StripQueryPlan {
    uint64_t uid = 0;
    int64_t nqp = 0;
    OwnedBuf pairs;
    Made made;
};

struct StripRefPlan {
    uint64_t uid = 0;
    int ngroups = 0;
    OwnedBuf buf;                    // meta, groups, slab
    const int2 *meta = nullptr, *groups = nullptr;
    const uint32_t* slab = nullptr;
    Made made;
};

std::vector<int32_t> longest_first(const st_seqset_s& s) {
    std::vector<int32_t> order(static_cast<size_t>(s.count)), at(size_t(s.max_len) + 2, 0);
    for (int32_t l : s.h_len) ++at[size_t(s.max_len - l) + 1];
    for (size_t l = 1; l < at.size(); ++l) at[l] += at[l - 1];
    for (int64_t i = 0; i < s.count; ++i) order[size_t(at[size_t(s.max_len - s.h_len[size_t(i)])]++)] = int32_t(i);
    return order;
}

template <class Plan>
Plan& strip_slot(std::shared_ptr<void>& own, std::shared_ptr<void>& shared, bool owns) {
    std::shared_ptr<void>& slot = owns ? own : shared;
    if (!slot) slot = std::make_shared<Plan>();
    return *static_cast<Plan*>(slot.get());
}

StripQueryPlan& query_plan(st_seqset_s& s, Context& ctx, cudaStream_t stream) {
    auto& p = strip_slot<StripQueryPlan>(s.strip_query_plan, ctx.tmp_strip_query_plan, s.owns);
    if (p.uid != s.uid) {
        std::vector<int32_t> order = longest_first(s);
        if (order.size() & 1) order.push_back(order.back());
        p.uid = 0;
        h2d(p.pairs.as<int32_t>(order.size(), stream), order.data(), order.size() * 4, stream);
        if (s.owns) p.made.on(stream);
        p.nqp = int64_t(order.size() / 2);
        p.uid = s.uid;
    }
    p.made.need(stream);
    return p;
}

StripRefPlan& ref_plan(st_seqset_s& s, Context& ctx, cudaStream_t stream) {
    auto& p = strip_slot<StripRefPlan>(s.strip_ref_plan, ctx.tmp_strip_ref_plan, s.owns);
    if (p.uid != s.uid) {
        const std::vector<int32_t> order = longest_first(s);
        const size_t ngroups = size_t(ceil_div(s.count, 32));
        std::vector<int2> up(order.size() + ngroups);  // meta, then groups
        for (size_t t = 0; t < order.size(); ++t) up[t] = make_int2(order[t], s.h_len[size_t(order[t])]);
        int64_t rows = 0;
        for (size_t g = 0; g < ngroups; ++g) {
            const int longest = up[g * 32].y;
            const bool one_length = g * 32 + 32 <= order.size() && up[g * 32 + 31].y == longest;
            up[order.size() + g] = make_int2(int(rows), longest | (one_length ? 1 << 16 : 0));
            rows += (longest + 3) / 4;
        }
        if (rows > INT32_MAX) fail(ST_EINVAL, "seqtree_b200: reference set too large for one call");
        p.uid = 0;
        const size_t slab_at = (up.size() * sizeof(int2) + 255) & ~size_t(255);
        uint8_t* d = p.buf.as<uint8_t>(slab_at + size_t(rows) * 128, stream);
        p.meta = reinterpret_cast<int2*>(d);
        p.groups = p.meta + order.size();
        auto* slab = reinterpret_cast<uint32_t*>(d + slab_at);
        p.slab = slab;
        h2d(d, up.data(), up.size() * sizeof(int2), stream);
        strip_slab_kernel<<<unsigned(ngroups), 256, 0, stream>>>(s.d_bytes, s.d_off, p.meta, s.count, p.groups, slab);
        STB_CUDA(cudaGetLastError());
        note_launch(nullptr);
        if (s.owns) p.made.on(stream);
        p.ngroups = int(ngroups);
        p.uid = s.uid;
    }
    p.made.need(stream);
    return p;
}

}  // namespace

bool strip_planned(const st_seqset_s& s, bool query) {
    if (!s.owns) return false;
    if (query) return s.strip_query_plan && static_cast<const StripQueryPlan*>(s.strip_query_plan.get())->uid == s.uid;
    return s.strip_ref_plan && static_cast<const StripRefPlan*>(s.strip_ref_plan.get())->uid == s.uid;
}

void strip_forget(st_seqset_s& s, bool query) {
    Context& ctx = context();
    if (query) {
        const auto& p = s.owns ? s.strip_query_plan : ctx.tmp_strip_query_plan;
        if (p) static_cast<StripQueryPlan*>(p.get())->uid = 0;
    } else {
        const auto& p = s.owns ? s.strip_ref_plan : ctx.tmp_strip_ref_plan;
        if (p) static_cast<StripRefPlan*>(p.get())->uid = 0;
    }
}

// Whether the strip kernel takes a call: gap_extend <= gap_open (the raised forms need it), no
// empty sequence, lengths up to 512, and every raised state of every real or padded cell within
// +-14000, so that int16 halves hold it (local mode adds kBias: 30384 < 32767).  Padding adds at
// most 64 rows (4 per strip) and 3 columns; |value| <= |s| * min(rows, cols) + open + extend *
// (rows + cols) in global mode, whose raise the last term counts, and less in local mode.
bool strip_eligible(const st_seqset_s& qs, const st_seqset_s& rs, const int32_t* sim, int A,
                    int32_t go, int32_t ge) {
    if (ge > go) return false;
    for (const st_seqset_s* s : {&qs, &rs}) {
        if (s->max_len > 512) return false;
        for (int32_t l : s->h_len)
            if (l < 1) return false;
    }
    int64_t maxabs = 0;
    for (int i = 0; i < A * A; ++i) maxabs = std::max<int64_t>(maxabs, std::llabs(int64_t(sim[i])));
    if (maxabs > 2000) return false;
    const int64_t rows = qs.max_len + 64, cols = rs.max_len + 4;
    return maxabs * (std::min(rows, cols) + 1) + 2 * int64_t(go) + int64_t(ge) * (rows + cols) <= 14000;
}

// Scores (or, with self scores, distances) of every pair into out_d; raised_d: s(a, b) + gap_extend in local
// mode, + 2 * gap_extend in global mode, on the device.
void align_strip(st_seqset_s& qs, st_seqset_s& rs, const int32_t* raised_d, int A, int32_t mode,
                 int32_t go, int32_t ge, int32_t dist, const int64_t* q_self, const int64_t* r_self,
                 int32_t* out_d, unsigned int* ovf, cudaStream_t stream) {
    Context& ctx = context();
    const bool local = mode == ST_MODE_LOCAL;
    const int add = local ? ge : 2 * ge;
    StripQueryPlan& qp = query_plan(qs, ctx, stream);
    StripRefPlan& rp = ref_plan(rs, ctx, stream);
    StripArgs a{};
    a.sim = raised_d;
    a.A = A;
    a.add = add;
    a.go = go;
    a.ge = ge;
    a.one = 1u;
    a.qc = qs.d_bytes;
    a.qoff = qs.d_off;
    a.qpairs = static_cast<const int2*>(qp.pairs.ptr);
    a.nqp = qp.nqp;
    a.slab = rp.slab;
    a.groups = rp.groups;
    a.rmeta = rp.meta;
    a.K = rs.count;
    a.ngroups = rp.ngroups;
    a.dist = dist;
    a.q_self = q_self;
    a.r_self = r_self;
    a.out = out_d;
    a.overflow = ovf;

    const int most = qs.max_len <= 32 ? 32 : 48;
    const void* kern =
        most == 48 ? (local ? reinterpret_cast<const void*>(gotoh_strip_kernel<48, true>)
                            : reinterpret_cast<const void*>(gotoh_strip_kernel<48, false>))
                   : (local ? reinterpret_cast<const void*>(gotoh_strip_kernel<32, true>)
                            : reinterpret_cast<const void*>(gotoh_strip_kernel<32, false>));
    int most_rows = 0;  // the tallest profile over the lengths up to the longest query
    for (int m = std::max(1, qs.max_len - most); m <= qs.max_len; ++m) {
        int strips, R;
        strip_shape(m, most, strips, R);
        most_rows = std::max(most_rows, strips * R);
    }
    const size_t smem = size_t(most_rows) * kProfW * 4;
    ensure_smem_limit(kern, smem);
    int per_sm = 0;
    STB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kStripWarps * 32, smem));
    const int64_t resident = int64_t(ctx.num_sms) * std::max(per_sm, 1);
    // Groups per warp and unit: enough columns to outweigh building the profile (a few thousand
    // cycles against about 8 per row and column), while every CTA still gets eight units.
    const int64_t cycles = int64_t(std::max(4, qs.max_len)) * std::max(4, rs.max_len) * 8;
    const int64_t want = std::max<int64_t>(1, 64000 / cycles);
    const int64_t room = std::max<int64_t>(1, a.nqp * rp.ngroups / (resident * kStripWarps * 8));
    a.gpw = int(std::min<int64_t>({want, room, ceil_div(rp.ngroups, kStripWarps)}));
    a.nchunks = int(ceil_div(rp.ngroups, int64_t(kStripWarps) * a.gpw));
    const int64_t grid = std::min<int64_t>(resident, a.nqp * a.nchunks);
    a.scratch_cols = qs.max_len > most ? ceil_div(rs.max_len, 4) * 4 : 0;
    const bool queued = grid < a.nqp * a.nchunks;
    const size_t columns = size_t(grid) * kStripWarps * size_t(a.scratch_cols) * 32 * sizeof(uint2);
    StreamScratch scratch(ctx.device, columns + (queued ? 256 : 0), stream);
    a.scratch = static_cast<uint2*>(scratch.ptr);
    if (queued) {
        a.queue = reinterpret_cast<unsigned long long*>(static_cast<uint8_t*>(scratch.ptr) + columns);
        STB_CUDA(cudaMemsetAsync(a.queue, 0, sizeof(unsigned long long), stream));
    }
    void* args[] = {&a};
    STB_CUDA(cudaLaunchKernel(kern, dim3(unsigned(grid)), dim3(kStripWarps * 32), args, smem, stream));
    note_launch("gotoh_strip_kernel");
}

}  // namespace stb
