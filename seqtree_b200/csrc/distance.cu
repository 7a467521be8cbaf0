// Dense Hamming and Levenshtein matrices over raw bytes (case-sensitive) on sm_100a.
//
// Reference: seqtree src/distance.cpp:68-109.  Both distances compare bytes for equality only,
// so a call maps the bytes present in either set to dense codes 0..sigma-1 (any bijection preserves
// equality; the table travels with the launch) and then:
//
//   Hamming (output-write bound): every string is packed at b = 1/2/4/8 bits per symbol into
//   32-bit words; a pair costs one XOR, one fold of each symbol's b bits onto its lowest bit and
//   one POPC per word.  A thread owns four consecutive columns and streams 16-byte stores, so a
//   warp writes 512 contiguous bytes of a row per query.
//
//   Levenshtein (integer-ALU bound): Myers' bit-vector algorithm in Hyyro's formulation for
//   whole-string edit distance.  The ref is the bit pattern (one integer of 1 to 16 32-bit words per
//   lane, as many as the longest ref needs) and the query is the text, warp-uniform, so the
//   per-character loop never diverges; the pattern-match masks Peq[c] of the 32 lanes live in
//   shared memory as [c][word][lane].  Lanes own 32 consecutive refs, so stores stay coalesced in
//   the original column order.  Longer refs, or more than 64 distinct symbols, take a
//   one-thread-per-pair DP with its row in global scratch (any length).
#include <algorithm>
#include <map>

#include "common.cuh"

namespace stb {

namespace {

// ------------------------------------------------------------------------- alphabets -------
struct alignas(4) ByteLut {
    uint8_t v[256];
};

// Up to two sets' bytes in one launch, a set per blockIdx.y.
struct TwoSets {
    const uint8_t* in[2];
    int64_t bytes[2];
};

// Byte-presence bitmap of each set (distinct bytes -> dense codes).
__global__ void presence_kernel(const TwoSets t, unsigned int* __restrict__ present) {
    __shared__ unsigned int s[8];
    if (threadIdx.x < 8) s[threadIdx.x] = 0;
    __syncthreads();
    const uint8_t* bytes = t.in[blockIdx.y];
    const int64_t n = t.bytes[blockIdx.y];
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += int64_t(gridDim.x) * blockDim.x) {
        const uint8_t c = bytes[i];
        atomicOr(&s[c >> 5], 1u << (c & 31));
    }
    __syncthreads();
    if (threadIdx.x < 8 && s[threadIdx.x]) atomicOr(&present[blockIdx.y * 8 + threadIdx.x], s[threadIdx.x]);
}

// What a set keeps for the distances: which bytes it holds, and its dense codes (Levenshtein) and
// packed words (Hamming) under the alphabets it has met.  The alphabet of a call is the union of both
// sets' bytes.  Nothing here is ever written again once it is made, so calls on several streams and
// captured graphs may read it for as long as the set lives, whatever partners the set meets in
// between; an alphabet past the last place is coded for its call alone.
constexpr int kMaxKept = 8;  // of either kind

enum Form { kCodes, kWords };

struct Kept {
    Form form;
    uint32_t symbols[8];
    void* ptr;
    size_t bytes;
    std::shared_ptr<Made> made;
};

struct DistPlan {
    uint64_t uid = 0;               // set the plan was built for
    bool owns = true;               // false: a transient set's, in buffers that the next one takes over
    uint32_t present[8] = {};       // bytes of the set
    std::vector<Kept> kept;
    DevBuf transient[2];            // by form
    ~DistPlan() {  // (with the set, after its bytes: freeing those waits for the kernels that read either)
        for (const Kept& k : kept)
            if (owns) kept_free(k.ptr, k.bytes);
    }
};

struct Alphabet {
    uint32_t symbols[8];
    ByteLut lut;   // byte -> 0 .. sigma - 1
    int sigma;
};

DistPlan& dist_plan(st_seqset_s& s, Context& ctx, int slot) {
    std::shared_ptr<void>& holder = s.owns ? s.dist_plan : ctx.tmp_dist_plan[slot];
    if (!holder) {
        holder = std::make_shared<DistPlan>();
        static_cast<DistPlan*>(holder.get())->owns = s.owns;
    }
    return *static_cast<DistPlan*>(holder.get());
}

Alphabet joint_alphabet(st_seqset_s& a, st_seqset_s& b, DistPlan* const plans[2], cudaStream_t stream,
                        Context& ctx) {
    const st_seqset_s* sets[2] = {&a, &b};
    auto* present = reinterpret_cast<unsigned int*>(ctx.flags_d + 16);
    const auto* bits = reinterpret_cast<const unsigned int*>(ctx.flags_h + 16);
    if (plans[0]->uid != a.uid || plans[1]->uid != b.uid) {
        refuse_capture(stream);
        STB_CUDA(cudaMemsetAsync(present, 0, 64, stream));
        TwoSets args{};
        for (int t = 0; t < 2; ++t) {
            args.in[t] = sets[t]->d_bytes;
            args.bytes[t] = plans[t]->uid == sets[t]->uid ? 0 : sets[t]->total;
        }
        const int64_t most = std::max<int64_t>({args.bytes[0], args.bytes[1], 1});
        presence_kernel<<<dim3(unsigned(std::min<int64_t>(ceil_div(most, 256), ctx.num_sms * 4)), 2), 256, 0,
                          stream>>>(args, present);
        STB_CUDA(cudaGetLastError());
        note_launch(nullptr);
        STB_CUDA(cudaMemcpyAsync(ctx.flags_h + 16, present, 64, cudaMemcpyDeviceToHost, stream));
        STB_CUDA(cudaStreamSynchronize(stream));
        for (int t = 0; t < 2; ++t) {
            if (plans[t]->uid == sets[t]->uid) continue;
            std::memcpy(plans[t]->present, bits + 8 * t, 32);
            plans[t]->kept.clear();  // (empty but for a transient set's plan)
            plans[t]->uid = sets[t]->uid;
        }
    }
    Alphabet al;
    for (int w = 0; w < 8; ++w) al.symbols[w] = plans[0]->present[w] | plans[1]->present[w];
    std::memset(al.lut.v, 0, sizeof al.lut.v);
    al.sigma = 0;
    for (int c = 0; c < 256; ++c)
        if (al.symbols[c >> 5] & (1u << (c & 31))) al.lut.v[c] = uint8_t(al.sigma++);
    return al;
}

// Both sets' codes or packed words for one call: those they keep, or room for what the call makes.
struct CallForms {
    void* ptr[2] = {};
    int todo[2], count = 0;         // the sets whose form is to be made, with one launch on the call's stream
    StreamScratch fresh[2];
    size_t size[2];
    bool keep[2] = {};

    CallForms(Form form, const Alphabet& al, st_seqset_s* const sets[2], DistPlan* const plans[2],
              const size_t (&bytes)[2], cudaStream_t stream, Context& ctx)
        : size{bytes[0], bytes[1]} {
        for (int t = 0; t < 2; ++t) {
            if (t == 1 && sets[0] == sets[1]) {
                ptr[1] = ptr[0];
                break;
            }
            DistPlan& p = *plans[t];
            int have = 0;
            for (const Kept& k : p.kept) {
                have += k.form == form;
                if (k.form != form || std::memcmp(k.symbols, al.symbols, 32) != 0) continue;
                ptr[t] = k.ptr;
                k.made->need(stream);
            }
            if (ptr[t]) continue;
            keep[t] = !p.owns || have < kMaxKept;
            if (keep[t]) refuse_capture(stream);
            if (p.owns) {
                fresh[t].take(ctx.device, std::max<size_t>(bytes[t], 16), stream, keep[t]);
                ptr[t] = fresh[t].ptr;
            } else {
                ptr[t] = p.transient[form].get(bytes[t]);
            }
            todo[count++] = t;
        }
    }
    // After the launch (nothing is kept of a call that fails before).
    void made(Form form, const Alphabet& al, DistPlan* const plans[2], cudaStream_t stream) {
        for (int t = 0; t < 2; ++t) {
            if (!keep[t]) continue;
            Kept k{form, {}, ptr[t], size[t], std::make_shared<Made>()};
            std::memcpy(k.symbols, al.symbols, 32);
            if (plans[t]->owns) k.made->on(stream);
            plans[t]->kept.push_back(std::move(k));
            fresh[t].keep();
        }
    }
};

// The table in shared memory (every thread of a block of at least 64 calls this).
__device__ __forceinline__ void load_lut(uint8_t* s, const ByteLut& lut) {
    if (threadIdx.x < 64)
        reinterpret_cast<uint32_t*>(s)[threadIdx.x] = reinterpret_cast<const uint32_t*>(lut.v)[threadIdx.x];
    __syncthreads();
}

// Dense codes of up to two sets' bytes, a set per blockIdx.y.
struct RemapArgs {
    const uint8_t* in[2];
    uint8_t* out[2];
    int64_t bytes[2];
};

__global__ void remap_kernel(const __grid_constant__ RemapArgs a, const __grid_constant__ ByteLut lut) {
    __shared__ __align__(4) uint8_t code[256];
    load_lut(code, lut);
    const uint8_t* in = a.in[blockIdx.y];
    uint8_t* out = a.out[blockIdx.y];
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < a.bytes[blockIdx.y];
         i += int64_t(gridDim.x) * blockDim.x)
        out[i] = code[in[i]];
}

// ---------------------------------------------------------------------------- Hamming -------
// Pack each string's codes (lut of its bytes) at B bits per symbol into W words (low symbol in low bits); up to two
// sets in one launch, a set per blockIdx.y.
struct PackArgs {
    const uint8_t* bytes[2];
    const int64_t* off[2];
    int64_t count[2];
    uint32_t* packed[2];
};

__global__ void pack_kernel(const __grid_constant__ PackArgs a, const __grid_constant__ ByteLut lut, int L, int B,
                            int W) {
    __shared__ __align__(4) uint8_t code[256];
    load_lut(code, lut);
    const int64_t s = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (s >= a.count[blockIdx.y]) return;
    const uint8_t* c = a.bytes[blockIdx.y] + a.off[blockIdx.y][s];
    const int per = 32 / B;
    for (int w = 0; w < W; ++w) {
        uint32_t v = 0;
        for (int t = 0; t < per; ++t) {
            const int j = w * per + t;
            if (j < L) v |= uint32_t(code[c[j]]) << (t * B);
        }
        a.packed[blockIdx.y][s * W + w] = v;
    }
}

template <int B>
__device__ __forceinline__ uint32_t fold_diff(uint32_t x) {
    if constexpr (B == 1) return x;
    if constexpr (B == 2) return (x | (x >> 1)) & 0x55555555u;
    if constexpr (B == 4) {
        x |= x >> 1;
        x |= x >> 2;
        return x & 0x11111111u;
    }
    x |= x >> 1;
    x |= x >> 2;
    x |= x >> 4;
    return x & 0x01010101u;
}

constexpr int kHamCols = 1024;  // columns per CTA (256 threads x 4)
constexpr int kHamRows = 32;    // query rows per CTA

template <int B, int W>
__global__ void __launch_bounds__(256) hamming_kernel(const uint32_t* __restrict__ qp,
                                                      const uint32_t* __restrict__ rp,
                                                      int64_t N, int64_t K,
                                                      int32_t* __restrict__ out) {
    const int64_t c0 = int64_t(blockIdx.x) * kHamCols + threadIdx.x * 4;
    const int64_t r0 = int64_t(blockIdx.y) * kHamRows;
    const int64_t r1 = (N < r0 + kHamRows ? N : r0 + kHamRows);
    if (c0 >= K) return;
    uint32_t rw[4][W];
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int w = 0; w < W; ++w) rw[t][w] = (c0 + t < K) ? __ldg(rp + (c0 + t) * W + w) : 0u;
    const bool full = (c0 + 4 <= K) && ((K & 3) == 0);
    for (int64_t i = r0; i < r1; ++i) {
        uint32_t qw[W];
#pragma unroll
        for (int w = 0; w < W; ++w) qw[w] = __ldg(qp + i * W + w);
        int v[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            int s = 0;
#pragma unroll
            for (int w = 0; w < W; ++w) s += __popc(fold_diff<B>(qw[w] ^ rw[t][w]));
            v[t] = s;
        }
        int32_t* dst = out + i * K + c0;
        if (full) {
            __stcs(reinterpret_cast<int4*>(dst), make_int4(v[0], v[1], v[2], v[3]));
        } else {
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if (c0 + t < K) dst[t] = v[t];
        }
    }
}

// Any word count: same scheme with the words read from memory.
template <int B>
__global__ void __launch_bounds__(256) hamming_kernel_any(const uint32_t* __restrict__ qp,
                                                          const uint32_t* __restrict__ rp,
                                                          int64_t N, int64_t K, int W,
                                                          int32_t* __restrict__ out) {
    const int64_t total = N * K;
    for (int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; idx < total;
         idx += int64_t(gridDim.x) * blockDim.x) {
        const int64_t i = idx / K, k = idx - i * K;
        int s = 0;
        for (int w = 0; w < W; ++w) s += __popc(fold_diff<B>(qp[i * W + w] ^ rp[k * W + w]));
        out[idx] = s;
    }
}

template <int B>
const char* launch_hamming(const uint32_t* qp, const uint32_t* rp, int64_t N, int64_t K, int W,
                           int32_t* out, cudaStream_t stream, int sms) {
    const dim3 grid(unsigned(ceil_div(K, kHamCols)), unsigned(ceil_div(N, kHamRows)));
    const bool tiled = grid.y <= 65535;
#define STB_HAM(WW)                                                                 \
    if (tiled && W == WW) {                                                         \
        hamming_kernel<B, WW><<<grid, 256, 0, stream>>>(qp, rp, N, K, out);         \
        STB_CUDA(cudaGetLastError());                                               \
        return "hamming_kernel";                                                    \
    }
    STB_HAM(1) STB_HAM(2) STB_HAM(3) STB_HAM(4) STB_HAM(6) STB_HAM(8)
#undef STB_HAM
    const int64_t blocks = std::min<int64_t>(ceil_div(N * K, 256), int64_t(sms) * 16);
    hamming_kernel_any<B><<<unsigned(blocks), 256, 0, stream>>>(qp, rp, N, K, W, out);
    STB_CUDA(cudaGetLastError());
    return "hamming_kernel_any";
}

// ---------------------------------------------------------------------------- Levenshtein ---
constexpr int kLevWarps = 8;

// s = a + b + carry over N = 2 or 4 words as one carry chain; `carry` (0 or 1) becomes the carry out.
template <int N>
__device__ __forceinline__ void add_words(uint32_t* s, const uint32_t* a, const uint32_t* b, uint32_t& carry) {
    static_assert(N == 2 || N == 4, "chains of two or four words");
    if constexpr (N == 2)
        asm("{ .reg .u32 x; add.cc.u32 x, %2, 0xffffffff; addc.cc.u32 %0, %3, %5; addc.cc.u32 %1, %4, %6;"
            " addc.u32 %2, 0, 0; }"
            : "=&r"(s[0]), "=&r"(s[1]), "+r"(carry)
            : "r"(a[0]), "r"(a[1]), "r"(b[0]), "r"(b[1]));
    else
        asm("{ .reg .u32 x; add.cc.u32 x, %4, 0xffffffff; addc.cc.u32 %0, %5, %9; addc.cc.u32 %1, %6, %10;"
            " addc.cc.u32 %2, %7, %11; addc.cc.u32 %3, %8, %12; addc.u32 %4, 0, 0; }"
            : "=&r"(s[0]), "=&r"(s[1]), "=&r"(s[2]), "=&r"(s[3]), "+r"(carry)
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]));
}

// s = a + b over NW words (the carry out of the last word is dropped).
template <int NW>
__device__ __forceinline__ void add_all(uint32_t* s, const uint32_t* a, const uint32_t* b) {
    if constexpr (NW == 1) {
        s[0] = a[0] + b[0];
    } else if constexpr (NW == 2) {
        asm("add.cc.u32 %0, %2, %4; addc.u32 %1, %3, %5;"
            : "=&r"(s[0]), "=r"(s[1])
            : "r"(a[0]), "r"(a[1]), "r"(b[0]), "r"(b[1]));
    } else if constexpr (NW == 3) {
        asm("add.cc.u32 %0, %3, %6; addc.cc.u32 %1, %4, %7; addc.u32 %2, %5, %8;"
            : "=&r"(s[0]), "=&r"(s[1]), "=r"(s[2])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(b[0]), "r"(b[1]), "r"(b[2]));
    } else if constexpr (NW == 4) {
        asm("add.cc.u32 %0, %4, %8; addc.cc.u32 %1, %5, %9; addc.cc.u32 %2, %6, %10; addc.u32 %3, %7, %11;"
            : "=&r"(s[0]), "=&r"(s[1]), "=&r"(s[2]), "=r"(s[3])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]));
    } else {  // chains of four words (and two), each handing its carry on through a register
        static_assert(NW % 2 == 0, "whole chains");
        uint32_t carry = 0;
#pragma unroll
        for (int w = 0; w + 4 <= NW; w += 4) add_words<4>(s + w, a + w, b + w, carry);
        if constexpr (NW % 4 == 2) add_words<2>(s + NW - 2, a + NW - 2, b + NW - 2, carry);
    }
}

// Pattern = ref (lane), text = query (warp-uniform).  Peq in shared memory as [c][word][lane].  The
// pattern is one integer of NW 32-bit words: the add and the two shifts run across the words, the
// rest word by word -- ten ALU operations a word and text character, whatever NW (a blocked form
// that hands each word's bottom step to the next costs eight more per 64 bits).  Rows past a lane's
// own ref length act as unmatched rows below the pattern and never reach rows above them, so every
// lane runs all NW words and masks its own length at the end.
// The bound is the ALU pipe.  Measured, B200: 20,000 x 20,000 ACGT 30-60 (NW 2) 21.5 -> 20.7
// ms (64-bit words, 16 rows per CTA -> this; ALU 88 %); 5,003 x 10,007 amino acids 8-25 (NW 1) 1.13 ->
// 0.60 ms (ALU 80 %, issue 79 %).
template <int NW>
__global__ void __launch_bounds__(kLevWarps * 32)
levenshtein_kernel(const uint8_t* __restrict__ qc, const int64_t* __restrict__ qoff,
                   const uint8_t* __restrict__ rc, const int64_t* __restrict__ roff, int64_t N,
                   int64_t K, int sigma, int rows, int32_t* __restrict__ out) {
    extern __shared__ uint32_t s_peq[];  // [warp][sigma][NW][32]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t* peq = s_peq + size_t(warp) * sigma * NW * 32;
    const int64_t k = (int64_t(blockIdx.x) * kLevWarps + warp) * 32 + lane;
    const bool valid = k < K;
    const int64_t kk = valid ? k : (K - 1);
    const uint8_t* r = rc + roff[kk];
    const int n = int(roff[kk + 1] - roff[kk]);
    for (int c = 0; c < sigma * NW; ++c) peq[c * 32 + lane] = 0u;
    for (int j = 0; j < n; ++j) peq[(r[j] * NW + (j >> 5)) * 32 + lane] |= 1u << (j & 31);
    __syncwarp();
    const uint32_t* mine = peq + lane;
    const int64_t r0 = int64_t(blockIdx.y) * rows;
    const int64_t r1 = (N < r0 + rows ? N : r0 + rows);
    for (int64_t i = r0; i < r1; ++i) {
        const uint8_t* q = qc + qoff[i];
        const int m = int(qoff[i + 1] - qoff[i]);
        // Pv / Mv hold the +1 / -1 vertical steps of the current DP column.  The distance is
        // read once from the last column, D[n][m] = D[0][m] + sum of its steps
        // = m + popc(Pv) - popc(Mv) over the n pattern bits, instead of following the bottom
        // cell through every column (which costs about a fifth of the loop's instructions).
        uint32_t Pv[NW], Mv[NW];
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            Pv[w] = ~0u;
            Mv[w] = 0u;
        }
        auto step = [&](int c) {
            const uint32_t* e = mine + c * (NW * 32);
            uint32_t Eq[NW], t[NW], Ph[NW], Mh[NW];
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                Eq[w] = e[w * 32];
                t[w] = Eq[w] & Pv[w];
            }
            add_all<NW>(t, t, Pv);
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                const uint32_t Xh = (t[w] ^ Pv[w]) | Eq[w];
                Ph[w] = Mv[w] | ~(Xh | Pv[w]);
                Mh[w] = Pv[w] & Xh;
            }
#pragma unroll
            for (int w = NW - 1; w >= 0; --w) {  // row 0 of the global distance: +1 per character
                const uint32_t Xv = Eq[w] | Mv[w];
                const uint32_t ph = w ? __funnelshift_l(Ph[w ? w - 1 : 0], Ph[w], 1) : Ph[0] * 2u + 1u;
                const uint32_t mh = w ? __funnelshift_l(Mh[w ? w - 1 : 0], Mh[w], 1) : Mh[0] * 2u;
                Pv[w] = mh | ~(Xv | ph);
                Mv[w] = ph & Xv;
            }
        };
        int t = 0;
        for (; t + 4 <= m; t += 4) {
            int c[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) c[u] = q[t + u];
#pragma unroll
            for (int u = 0; u < 4; ++u) step(c[u]);
        }
        for (; t < m; ++t) step(q[t]);
        int score = m;
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            const int bits = min(32, max(0, n - 32 * w));
            const uint32_t mask = bits >= 32 ? ~0u : (1u << bits) - 1u;
            score += __popc(Pv[w] & mask) - __popc(Mv[w] & mask);
        }
        if (valid) out[i * K + k] = score;
    }
}

using LevKernel = void (*)(const uint8_t*, const int64_t*, const uint8_t*, const int64_t*, int64_t, int64_t, int,
                           int, int32_t*);

// The kernel for refs of up to `longest` symbols and its words per pattern; null past 512 symbols.
LevKernel lev_kernel(int longest, int& words) {
    struct Form {
        int words;
        LevKernel kernel;
    };
    static const Form forms[] = {{1, levenshtein_kernel<1>},   {2, levenshtein_kernel<2>},
                                 {3, levenshtein_kernel<3>},   {4, levenshtein_kernel<4>},
                                 {6, levenshtein_kernel<6>},   {8, levenshtein_kernel<8>},
                                 {12, levenshtein_kernel<12>}, {16, levenshtein_kernel<16>}};
    for (const Form& f : forms)
        if (longest <= 32 * f.words) {
            words = f.words;
            return f.kernel;
        }
    words = 0;
    return nullptr;
}

// Any lengths / alphabets: classic single-row DP per (i, k), row kept in global scratch laid
// out [j][thread] so that neighbouring threads touch neighbouring words.
__global__ void __launch_bounds__(256)
levenshtein_dp_kernel(const uint8_t* __restrict__ qc, const int64_t* __restrict__ qoff,
                      const uint8_t* __restrict__ rc, const int64_t* __restrict__ roff, int64_t N,
                      int64_t K, int32_t* __restrict__ scratch, int32_t* __restrict__ out) {
    const int64_t T = int64_t(gridDim.x) * blockDim.x;
    const int64_t tid = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    for (int64_t idx = tid; idx < N * K; idx += T) {
        const int64_t i = idx / K, k = idx - i * K;
        const uint8_t* a = qc + qoff[i];
        const uint8_t* b = rc + roff[k];
        int m = int(qoff[i + 1] - qoff[i]), n = int(roff[k + 1] - roff[k]);
        if (n > m) {  // row over the shorter string (src/distance.cpp:80)
            const uint8_t* t = a; a = b; b = t;
            int u = m; m = n; n = u;
        }
        int32_t v;
        if (n == 0) {
            v = m;
        } else {
            for (int j = 0; j <= n; ++j) scratch[j * T + tid] = j;
            for (int x = 1; x <= m; ++x) {
                int diag = scratch[tid];
                int left = x;
                scratch[tid] = x;
                const uint8_t ax = a[x - 1];
                for (int j = 1; j <= n; ++j) {
                    const int up = scratch[j * T + tid];
                    const int cur = min(min(up + 1, left + 1), diag + (ax == b[j - 1] ? 0 : 1));
                    diag = up;
                    left = cur;
                    scratch[j * T + tid] = cur;
                }
            }
            v = scratch[n * T + tid];
        }
        out[idx] = v;
    }
}

}  // namespace

void hamming_sets(st_seqset_s& a, st_seqset_s& b, int32_t* out_d, cudaStream_t stream) {
    if (a.alphabet != -1 || b.alphabet != -1)
        fail(ST_EINVAL, "seqtree_b200: distance sets must hold raw bytes (alphabet -1)");
    const int64_t N = a.count, K = b.count;
    if (N == 0 || K == 0) return;
    // Every pair must have equal length (src/distance.cpp:68-72).  Report the first mismatched
    // pair in row-major order, as a one-thread reference run would.
    const int32_t L = a.h_len[0];
    int64_t bi = -1, bk = -1;
    bool refs_uniform = true;
    for (int64_t k = 0; k < K; ++k)
        if (b.h_len[size_t(k)] != b.h_len[0]) { refs_uniform = false; break; }
    if (!refs_uniform) {
        for (int64_t k = 0; k < K; ++k)
            if (b.h_len[size_t(k)] != L) { bi = 0; bk = k; break; }
    } else {
        for (int64_t i = 0; i < N; ++i)
            if (a.h_len[size_t(i)] != b.h_len[0]) { bi = i; bk = 0; break; }
    }
    if (bi >= 0)
        fail(ST_EINVAL, "seqtree: hamming distance is only defined for equal-length sequences (got " +
                            std::to_string(a.h_len[size_t(bi)]) + " and " +
                            std::to_string(b.h_len[size_t(bk)]) + ")");
    Context& ctx = context();
    st_seqset_s* sets[2] = {&a, &b};
    DistPlan* plans[2] = {&dist_plan(a, ctx, 0), &dist_plan(b, ctx, 1)};
    const Alphabet al = joint_alphabet(a, b, plans, stream, ctx);
    const int sigma = al.sigma;
    const int B = sigma <= 2 ? 1 : sigma <= 4 ? 2 : sigma <= 16 ? 4 : 8;
    const int per = 32 / B;
    const int W = std::max(1, int(ceil_div(L, per)));
    const size_t bytes[2] = {size_t(N) * size_t(W) * 4, size_t(K) * size_t(W) * 4};
    CallForms f(kWords, al, sets, plans, bytes, stream, ctx);
    if (f.count) {
        PackArgs pa{};
        for (int i = 0; i < f.count; ++i) {
            const st_seqset_s& s = *sets[f.todo[i]];
            pa.bytes[i] = s.d_bytes;
            pa.off[i] = s.d_off;
            pa.count[i] = s.count;
            pa.packed[i] = static_cast<uint32_t*>(f.ptr[f.todo[i]]);
        }
        const int64_t most = std::max(pa.count[0], pa.count[1]);
        pack_kernel<<<dim3(unsigned(ceil_div(most, 256)), unsigned(f.count)), 256, 0, stream>>>(pa, al.lut, L, B, W);
        STB_CUDA(cudaGetLastError());
        note_launch(nullptr);
        f.made(kWords, al, plans, stream);
    }
    const auto *qp = static_cast<const uint32_t*>(f.ptr[0]), *rp = static_cast<const uint32_t*>(f.ptr[1]);
    const char* name;
    switch (B) {
        case 1: name = launch_hamming<1>(qp, rp, N, K, W, out_d, stream, ctx.num_sms); break;
        case 2: name = launch_hamming<2>(qp, rp, N, K, W, out_d, stream, ctx.num_sms); break;
        case 4: name = launch_hamming<4>(qp, rp, N, K, W, out_d, stream, ctx.num_sms); break;
        default: name = launch_hamming<8>(qp, rp, N, K, W, out_d, stream, ctx.num_sms); break;
    }
    note_launch(name);
}

void levenshtein_sets(st_seqset_s& a, st_seqset_s& b, int32_t* out_d, cudaStream_t stream,
                      int64_t r0, int64_t r1) {
    if (a.alphabet != -1 || b.alphabet != -1)
        fail(ST_EINVAL, "seqtree_b200: distance sets must hold raw bytes (alphabet -1)");
    if (r1 < 0) r1 = a.count;
    if (r0 < 0 || r0 > r1 || r1 > a.count) fail(ST_EINVAL, "seqtree_b200: bad row range");
    const int64_t N = r1 - r0, K = b.count;
    if (N == 0 || K == 0) return;
    Context& ctx = context();
    DistPlan* plans[2] = {&dist_plan(a, ctx, 0), &dist_plan(b, ctx, 1)};
    const Alphabet al = joint_alphabet(a, b, plans, stream, ctx);
    const int sigma = std::max(1, al.sigma);
    // rows [r0, r1): their offsets and their block of the result
    const int64_t* aoff = a.d_off + r0;
    out_d += r0 * K;
    // Bit-vector path: refs up to 512 symbols while the Peq table fits.  Rows per CTA: enough that
    // building the table (about as long as one row) does not show, while the GPU (eight CTAs
    // per SM) still gets six waves of CTAs.
    int words = 0;
    const LevKernel kern = lev_kernel(b.max_len, words);
    const size_t smem = size_t(kLevWarps) * sigma * std::max(words, 1) * 32 * 4;
    const int64_t colblocks = ceil_div(K, kLevWarps * 32);
    const int rows = int(std::min<int64_t>(
        128, std::max<int64_t>(16, N * colblocks / (int64_t(ctx.num_sms) * 8 * 6))));
    const dim3 grid(unsigned(colblocks), unsigned(std::min<int64_t>(ceil_div(N, rows), 65536)));
    if (kern && sigma <= 64 && smem <= size_t(200) * 1024 && grid.y <= 65535) {
        st_seqset_s* sets[2] = {&a, &b};
        const size_t bytes[2] = {size_t(a.total), size_t(b.total)};
        CallForms f(kCodes, al, sets, plans, bytes, stream, ctx);
        if (f.count) {
            RemapArgs ra{};
            for (int i = 0; i < f.count; ++i) {
                ra.in[i] = sets[f.todo[i]]->d_bytes;
                ra.out[i] = static_cast<uint8_t*>(f.ptr[f.todo[i]]);
                ra.bytes[i] = sets[f.todo[i]]->total;
            }
            const int64_t most = std::max<int64_t>({ra.bytes[0], ra.bytes[1], 1});
            remap_kernel<<<dim3(unsigned(std::min<int64_t>(ceil_div(most, 256), ctx.num_sms * 4)), unsigned(f.count)),
                           256, 0, stream>>>(ra, al.lut);
            STB_CUDA(cudaGetLastError());
            note_launch(nullptr);
            f.made(kCodes, al, plans, stream);
        }
        ensure_smem_limit(reinterpret_cast<const void*>(kern), smem);
        kern<<<grid, kLevWarps * 32, smem, stream>>>(static_cast<const uint8_t*>(f.ptr[0]), aoff,
                                                     static_cast<const uint8_t*>(f.ptr[1]), b.d_off, N, K, sigma,
                                                     rows, out_d);
        STB_CUDA(cudaGetLastError());
        note_launch("levenshtein_kernel");
        return;
    }
    const int shorter_max = std::min(a.max_len, b.max_len);
    const int longer_max = std::max(a.max_len, b.max_len);
    (void)longer_max;
    // Scratch: (shorter+1) words per resident thread, bounded to 2 GiB.
    int64_t threads = std::min<int64_t>(int64_t(ctx.num_sms) * 2048, N * K);
    const int64_t per = int64_t(shorter_max) + 1;
    threads = std::max<int64_t>(256, std::min<int64_t>(threads, (int64_t(1) << 29) / per));
    threads = ceil_div(threads, 256) * 256;
    ScratchTurn turn(ctx, stream);
    StreamScratch own;
    int32_t* scratch = turn.as<int32_t>(ctx.work_a, size_t(threads) * per, own);
    levenshtein_dp_kernel<<<unsigned(threads / 256), 256, 0, stream>>>(a.d_bytes, aoff, b.d_bytes, b.d_off, N, K,
                                                                       scratch, out_d);
    STB_CUDA(cudaGetLastError());
    note_launch("levenshtein_dp_kernel");
}

}  // namespace stb
