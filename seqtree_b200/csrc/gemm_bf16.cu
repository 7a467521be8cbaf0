// BF16 tensor-core GEMM with fp32 accumulation for the encoder's training layers:
// C (=, +=) op(A) op(B) with fp32 operands and result (the fp32 master weights and activations
// stay fp32; only the products run in bf16).
//
// Both operands are first packed into the tcgen05 K-major operand layout in bf16: blocks of 128
// rows x 64 k (16 KB), row r at r*128 bytes, the 16-byte unit u of a row at u ^ (r & 7) (the
// 128-byte swizzle), zero outside the matrix.  Packing absorbs the transposes (op(A) is A or
// A^T, the same for B); a matrix that takes part in two products, along its rows and along its columns,
// is packed once and read MN-major for the second (pack_matrix).  One CTA computes
// one 128 x 128 output tile over a range of K chunks: warp 0 bulk-copies A and B chunks through a
// 2-stage shared-memory ring (64 KB, so that three CTAs share an SM and one's epilogue overlaps
// another's loads: the layers are thin), one thread of warp 1 issues M=128 N=128 K=16 tcgen05.mma into a
// 128-column TMEM accumulator, and warps 2-5 (one TMEM lane quarter each) stage the tile in
// shared memory, from where all six warps store, add or atomically add (split K) it into C with
// coalesced writes.
// Every wait is bounded.
#include <cuda_bf16.h>

#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "gemm_bf16.cuh"
#include "tc.cuh"

namespace stb {

namespace {

constexpr int kGT = 128;                 // tile rows (M) and columns (N)
constexpr int kGK = 64;                  // K per chunk: one 128-byte swizzled row
constexpr int kGStages = 2;
constexpr int kGThreads = 192;
constexpr int kBlockB = kGT * kGK * 2;   // 16 KB
constexpr int kGSmBar = kGStages * 2 * kBlockB;
constexpr size_t kGSmem = size_t(kGSmBar) + 128 + 1024;

// One value of an operand's matrix, (row r, column c); callers check the ranges.
template <int KIND>
__device__ __forceinline__ float src_value(const PackSrc& s, int64_t r, int c) {
    if constexpr (KIND == PackSrc::kConv) {
        const int t = int(r & 31) + (c >> 7) - 1, L = s.lens[r >> 5];
        return (int(r & 31) < L && t >= 0 && t < L) ? s.x[(r + (c >> 7) - 1) * s.ld + (c & 127)] : 0.f;
    }
    const int64_t at = r * s.ld + c;
    if constexpr (KIND == PackSrc::kRelu) return s.y[at] > 0.f ? s.x[at] : 0.f;
    return s.x[at];
}

// Eight consecutive values (row r, columns c..c+7, c a multiple of 8) as two 16-byte loads.
template <int KIND>
__device__ __forceinline__ void src_eight(const PackSrc& s, int64_t r, int c, float (&v)[8]) {
    int64_t at = r * s.ld + c;
    if constexpr (KIND == PackSrc::kConv) {
        const int t = int(r & 31) + (c >> 7) - 1, L = s.lens[r >> 5];
        if (int(r & 31) >= L || t < 0 || t >= L) {
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = 0.f;
            return;
        }
        at = (r + (c >> 7) - 1) * s.ld + (c & 127);
    }
    const float4 a = *reinterpret_cast<const float4*>(s.x + at), b = *reinterpret_cast<const float4*>(s.x + at + 4);
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
    if constexpr (KIND == PackSrc::kRelu) {
        const float4 p = *reinterpret_cast<const float4*>(s.y + at), q = *reinterpret_cast<const float4*>(s.y + at + 4);
        const float y[8] = {p.x, p.y, p.z, p.w, q.x, q.y, q.z, q.w};
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = y[e] > 0.f ? v[e] : 0.f;
    }
}

__device__ __forceinline__ uint4 bf16_unit(const float (&v)[8]) {
    union {
        uint4 q;
        __nv_bfloat162 h[4];
    } pk;
#pragma unroll
    for (int e = 0; e < 4; ++e) pk.h[e] = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
    return pk.q;
}

// Packed operand: op[(tile * kchunks + chunk)][row][unit], value(i, k) = matrix(i, k) (rows of the
// matrix are the operand's rows).  One thread per 16-byte output unit, in output order: a warp
// reads four 256-byte row pieces and writes 512 contiguous bytes.  VEC: 16-byte loads (base and leading
// dimension aligned, K a multiple of 8).
template <int KIND, bool VEC>
__global__ void pack_rows_kernel(const PackSrc s, int rows, int K, int kchunks, int64_t units,
                                 uint8_t* __restrict__ op) {
    const int64_t pos = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (pos >= units) return;
    const int pu = int(pos & 7);
    const int64_t rowblk = pos >> 3;  // (tile * kchunks + chunk) * 128 + row
    const int row = int(rowblk & 127);
    const int64_t blk = rowblk >> 7;  // tile * kchunks + chunk
    const int chunk = int(blk % kchunks);
    const int64_t i = (blk / kchunks) * kGT + row;
    const int k0 = chunk * kGK + (pu ^ (row & 7)) * 8;
    float v[8];
    if (VEC && i < rows && k0 < K) {
        src_eight<KIND>(s, i, k0, v);
    } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = (!VEC && i < rows && k0 + e < K) ? src_value<KIND>(s, i, k0 + e) : 0.f;
    }
    *reinterpret_cast<uint4*>(op + pos * 16) = bf16_unit(v);
}

// The same, four passes of 32 rows over one 128 x 64 block after another (kSumTiles of them), with the
// matrix' column sums: a thread meets the same eight columns in each of its rows (row & 7 is fixed), so
// the sums stay in registers until the end.  Aligned as VEC.
constexpr int kSumTiles = 4;

template <int KIND>
__global__ void __launch_bounds__(256) pack_rows_sum_kernel(const PackSrc s, int rows, int cols, int tiles,
                                                            uint8_t* __restrict__ op) {
    __shared__ float part[32][kGK + 1];
    const int kchunks = cols / kGK, chunk = blockIdx.x % kchunks, t0 = blockIdx.x / kchunks * kSumTiles;
    const int pu = threadIdx.x & 7, r0 = threadIdx.x >> 3;
    const int u = pu ^ (r0 & 7);
    float sum[8] = {};
    for (int t = t0; t < min(t0 + kSumTiles, tiles); ++t) {
#pragma unroll
        for (int p = 0; p < kGT / 32; ++p) {
            const int row = p * 32 + r0;
            const int64_t i = int64_t(t) * kGT + row;
            float v[8] = {};
            if (i < rows) src_eight<KIND>(s, i, chunk * kGK + u * 8, v);
#pragma unroll
            for (int e = 0; e < 8; ++e) sum[e] += v[e];
            *reinterpret_cast<uint4*>(op + (int64_t(t) * kchunks + chunk) * kBlockB + row * 128 + pu * 16) = bf16_unit(v);
        }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) part[r0][u * 8 + e] = sum[e];
    __syncthreads();
    if (threadIdx.x < kGK) {
        float total = 0.f;
#pragma unroll 8
        for (int r = 0; r < 32; ++r) total += part[r][threadIdx.x];
        atomicAdd(s.colsum + chunk * kGK + threadIdx.x, total);
    }
}

// A thread per 16-byte unit of any of the weights: one launch for the ten operands of a step, where each took
// one of 5 to 6 us by itself (2,048 pairs, B200: 2.05 -> 2.036 ms, device time 1,820 -> 1,763 us).
struct WeightArgs {
    WeightSrc w[kMaxWeights];
    int64_t unit0[kMaxWeights + 1];
    uint8_t* op;
};

__global__ void pack_weights_kernel(const __grid_constant__ WeightArgs a, int n) {
    const int64_t pos = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (pos >= a.unit0[n]) return;
    int i = 0;
    while (pos >= a.unit0[i + 1]) ++i;
    const WeightSrc& w = a.w[i];
    const int64_t at = pos - a.unit0[i];
    const int pu = int(at & 7), row = int(at >> 3) & (kGT - 1);
    const int64_t blk = at >> 10;  // tile * kchunks + chunk
    const int kchunks = w.cols / kGK;
    const int64_t r = blk / kchunks * kGT + row, c = blk % kchunks * kGK + (pu ^ (row & 7)) * 8;
    float v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = w.trans ? w.x[(c + e) * w.ld + r] : w.x[r * w.ld + c + e];
    *reinterpret_cast<uint4*>(a.op + pos * 16) = bf16_unit(v);
}

// The same packed operand from the transpose: value(i, k) = matrix(k, i).  One 256-thread
// block per (tile, chunk) block: it reads the 64 x 128 fp32 piece row by row (coalesced)
// into shared memory and writes the 16 KB block in output order.
__global__ void __launch_bounds__(256) pack_cols_kernel(const PackSrc s, int rows, int K, int kchunks,
                                                        uint8_t* __restrict__ op) {
    __shared__ float t[kGK][kGT + 1];
    const int chunk = int(blockIdx.x % unsigned(kchunks));
    const int64_t i0 = int64_t(blockIdx.x / unsigned(kchunks)) * kGT;
    const int k0 = chunk * kGK;
#pragma unroll 8
    for (int idx = threadIdx.x; idx < kGK * kGT; idx += 256) {
        const int kk = idx >> 7, ii = idx & 127;
        const int64_t i = i0 + ii;
        t[kk][ii] = (i < rows && k0 + kk < K) ? src_value<PackSrc::kPlain>(s, k0 + kk, int(i)) : 0.f;
    }
    __syncthreads();
    uint8_t* dst = op + int64_t(blockIdx.x) * kBlockB;
#pragma unroll
    for (int pos = threadIdx.x; pos < kGT * 8; pos += 256) {
        const int row = pos >> 3, u = (pos & 7) ^ (row & 7);
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = t[u * 8 + e][row];
        *reinterpret_cast<uint4*>(dst + pos * 16) = bf16_unit(v);
    }
}

struct GemmBf16Args {
    const uint8_t* a;   // packed op(A): mtiles x kchunks blocks
    const uint8_t* b;   // packed op(B): ntiles x kchunks blocks
    int kchunks, chunks_per_split;
    int acols, bcols;   // TN: 64-column blocks of a row of A and of B
    float* C;
    int ldc, M, N;
    int mode;           // 0 store, 1 add, 2 atomic add
    GemmEpi epi;        // (mode 0 or 1)
    unsigned long long* err;
};

// MN-major operand in the 128-byte swizzle: 64 columns x 8 k to an atom of 1024 B, the next 8 k 1024 B on
// and the next 64 columns kBlockB / 2 on.
__device__ __forceinline__ uint64_t sw128_desc_mn(uint32_t addr) {
    return uint64_t((addr >> 4) & 0x3FFFu) | (uint64_t(kBlockB / 2 >> 4) << 16) | (uint64_t(1024 >> 4) << 32) |
           (uint64_t(1) << 46) | (uint64_t(2) << 61);
}

// TN: C = A^T B of two matrices packed as rows: a chunk is 64 of their rows, two half blocks (64 columns each)
// of either, read MN-major.  Packing both transposes instead took 503 us of a 2,048-pair step.
template <bool TN>
__global__ void __launch_bounds__(kGThreads) gemm_bf16_kernel(GemmBf16Args g) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((uintptr_t(smem_raw) + 1023) & ~uintptr_t(1023));
    // barriers: 0-1 full, 2-3 empty, 6 accumulator ready, 7 MMA drain
    const uint32_t bar0 = smem_u32(smem + kGSmBar);
    auto BAR = [&](int i) { return bar0 + 8u * uint32_t(i); };
    uint32_t* s_tmem = reinterpret_cast<uint32_t*>(smem + kGSmBar + 64);
    volatile int* s_abort = reinterpret_cast<volatile int*>(smem + kGSmBar + 68);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tn = blockIdx.x, tm = blockIdx.y;
    const int c0 = blockIdx.z * g.chunks_per_split;
    const int c1 = min(g.kchunks, c0 + g.chunks_per_split);
    if (threadIdx.x == 0) {
        for (int s = 0; s < kGStages; ++s) {
            bar_init(BAR(s), 1);
            bar_init(BAR(kGStages + s), 1);
        }
        bar_init(BAR(6), 1);
        bar_init(BAR(7), 1);
        *s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    if (warp == 1) tmem_alloc(smem_u32(s_tmem), 128);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *s_tmem;
    const uint32_t sbase = smem_u32(smem);

    if (warp == 0 && lane == 0) {
        uint32_t stage = 0, phase = 0, issued = 0, par = 0;
        for (int c = c0; c < c1; ++c) {
            if (!bar_wait(BAR(kGStages + stage), phase ^ 1u, s_abort, g.err)) break;
            bar_expect_tx(BAR(stage), 2 * kBlockB);
            const uint32_t dst = sbase + stage * 2 * kBlockB;
            if (TN) {
                const int64_t half = int64_t(c & 1) * (kBlockB / 2);
                for (int j = 0; j < 2; ++j) {
                    bulk_load(dst + j * (kBlockB / 2), g.a + (int64_t(c >> 1) * g.acols + 2 * tm + j) * kBlockB + half,
                              kBlockB / 2, BAR(stage));
                    bulk_load(dst + kBlockB + j * (kBlockB / 2),
                              g.b + (int64_t(c >> 1) * g.bcols + 2 * tn + j) * kBlockB + half, kBlockB / 2, BAR(stage));
                }
            } else {
                bulk_load(dst, g.a + (int64_t(tm) * g.kchunks + c) * kBlockB, kBlockB, BAR(stage));
                bulk_load(dst + kBlockB, g.b + (int64_t(tn) * g.kchunks + c) * kBlockB, kBlockB, BAR(stage));
            }
            issued |= 1u << stage;
            par = phase ? (par | (1u << stage)) : (par & ~(1u << stage));
            if (++stage == kGStages) {
                stage = 0;
                phase ^= 1u;
            }
        }
        for (int s = 0; s < kGStages; ++s)
            if (issued & (1u << s)) bar_drain(BAR(s), (par >> s) & 1u);
    } else if (warp == 1 && lane == 0) {
        constexpr uint32_t idesc = idesc_bf16(128, 128) | (TN ? 3u << 15 : 0u);  // A and B MN-major
        uint32_t stage = 0, phase = 0;
        for (int c = c0; c < c1; ++c) {
            if (!bar_wait(BAR(stage), phase, s_abort, g.err)) break;
            tc_fence_after();
            const uint32_t a = sbase + stage * 2 * kBlockB, b = a + kBlockB;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
                tc_mma(tmem, TN ? sw128_desc_mn(a + kk * 2048) : sw128_desc(a + kk * 32),
                       TN ? sw128_desc_mn(b + kk * 2048) : sw128_desc(b + kk * 32), idesc,
                       (c > c0 || kk > 0) ? 1u : 0u);
            tc_commit(BAR(kGStages + stage));
            if (++stage == kGStages) {
                stage = 0;
                phase ^= 1u;
            }
        }
        tc_commit(BAR(6));
        tc_commit(BAR(7));
        bar_drain(BAR(7), 0);
    } else if (warp >= 2) {
        const int quarter = warp & 3;
        if (c1 > c0 && bar_wait_own(BAR(6), 0, g.err)) {
            tc_fence_after();
            // The warp's 32 x 128 fp32 quarter goes to the (now idle) ring: TMEM lane r -> tile
            // row quarter * 32 + r, its 16-byte unit u at u ^ (r & 7) (conflict-free both ways).
            float* stage = reinterpret_cast<float*>(smem + quarter * (32 * kGT * 4));
            const uint32_t tl = tmem + (uint32_t(quarter * 32) << 16);
#pragma unroll 1
            for (int grp = 0; grp < 4; ++grp) {
                uint32_t v[32];
                __syncwarp();
                tmem_ld32(tl + uint32_t(grp * 32), v);
#pragma unroll
                for (int t = 0; t < 8; ++t)
                    *reinterpret_cast<uint4*>(stage + lane * kGT + (((grp * 8 + t) ^ (lane & 7)) << 2)) =
                        make_uint4(v[4 * t], v[4 * t + 1], v[4 * t + 2], v[4 * t + 3]);
            }
        } else {
            *s_abort = 1;
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        tmem_free(tmem, 128);
    }
    if (c1 <= c0 || *s_abort) return;
    // All six warps write the staged tile out, a warp per row at a time (128 consecutive
    // columns per instruction), four rows per batch so that the loads of the add mode overlap.
    const float* stage = reinterpret_cast<const float*>(smem);
    constexpr int kWarps = kGThreads / 32;
#pragma unroll 1
    for (int r0 = warp; r0 < kGT; r0 += 4 * kWarps) {
        float x[4][4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int r = r0 + b * kWarps;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int c = lane + 32 * q;
                x[b][q] = r < kGT ? stage[r * kGT + (((c >> 2) ^ (r & 7)) << 2) + (c & 3)] : 0.f;
            }
        }
        const GemmEpi& ep = g.epi;
        const float* addend = ep.kind == GemmEpi::kResidual || ep.kind == GemmEpi::kConv ? ep.res
                              : g.mode == 1                                              ? g.C
                                                                                         : nullptr;
        float y[4][4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int r = r0 + b * kWarps, row = tm * kGT + r;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int col = tn * kGT + lane + 32 * q;
                y[b][q] = (addend && r < kGT && row < g.M && col < g.N) ? addend[int64_t(row) * g.ldc + col] : 0.f;
            }
        }
        float bias[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int col = tn * kGT + lane + 32 * q;
            bias[q] = ep.bias && col < g.N ? ep.bias[col] : 0.f;
        }
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int r = r0 + b * kWarps, row = tm * kGT + r;
            if (r >= kGT || row >= g.M) continue;
            const bool valid = !ep.lens || (row & 31) < ep.lens[row >> 5];
            float* crow = g.C + int64_t(row) * g.ldc;
            float* orow = ep.out + int64_t(row) * g.ldc;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int col = tn * kGT + lane + 32 * q;
                if (col >= g.N) continue;
                // (the sums in the order of the separate passes they replace)
                switch (ep.kind) {
                    case GemmEpi::kBias: crow[col] = x[b][q] + bias[q]; break;
                    case GemmEpi::kResidual: orow[col] = valid ? y[b][q] + x[b][q] + bias[q] : 0.f; break;
                    case GemmEpi::kConv: {
                        const float p = x[b][q] + bias[q];
                        crow[col] = p;
                        orow[col] = valid ? y[b][q] + fmaxf(p, 0.f) : 0.f;
                        break;
                    }
                    case GemmEpi::kMaskAdd: crow[col] = valid ? x[b][q] + y[b][q] : 0.f; break;
                    default:
                        if (g.mode == 2) atomicAdd(crow + col, x[b][q]);
                        else crow[col] = g.mode == 1 ? x[b][q] + y[b][q] : x[b][q];
                }
            }
        }
    }
}

bool vec_ok(const PackSrc& s, int K) {
    return ((uintptr_t(s.x) | uintptr_t(s.y)) & 15) == 0 && s.ld % 4 == 0 && K % 8 == 0;
}

// op[i][k] = trans ? s[k][i] : s[i][k]
size_t pack_bytes(int rows, int K) { return size_t(ceil_div(rows, kGT)) * size_t(ceil_div(K, kGK)) * kBlockB; }

const uint8_t* pack(const PackSrc& s, bool trans, int rows, int K, uint8_t* op, cudaStream_t st) {
    const int tiles = int(ceil_div(rows, kGT)), kchunks = int(ceil_div(K, kGK));
    const int64_t units = int64_t(tiles) * kchunks * kGT * 8;
    if (trans)
        pack_cols_kernel<<<unsigned(tiles * kchunks), 256, 0, st>>>(s, rows, K, kchunks, op);
    else
        (vec_ok(s, K) ? pack_rows_kernel<PackSrc::kPlain, true> : pack_rows_kernel<PackSrc::kPlain, false>)
            <<<unsigned(ceil_div(units, 256)), 256, 0, st>>>(s, rows, K, kchunks, units, op);
    STB_CUDA(cudaGetLastError());
    return op;
}

template <int KIND>
void launch_matrix(const PackSrc& s, int rows, int cols, int tiles, uint8_t* op, cudaStream_t st) {
    const int kchunks = cols / kGK;
    const int64_t units = int64_t(tiles) * kchunks * kGT * 8;
    if (s.colsum)
        pack_rows_sum_kernel<KIND><<<unsigned(ceil_div(tiles, kSumTiles)) * kchunks, 256, 0, st>>>(s, rows, cols, tiles, op);
    else
        pack_rows_kernel<KIND, true><<<unsigned(ceil_div(units, 256)), 256, 0, st>>>(s, rows, cols, kchunks, units, op);
}

// The product of packed operands.  Products with a long K and few output tiles are split over K and added
// atomically, in which case C must already hold the value to add to (it is cleared first when
// !accumulate).  An epilogue other than kNone takes the product unsplit.
void run_gemm(GemmBf16Args g, bool tn, bool accumulate, cudaStream_t st, int sms) {
    Context& ctx = context();
    const int mtiles = int(ceil_div(g.M, kGT)), ntiles = int(ceil_div(g.N, kGT)), tiles = mtiles * ntiles;
    int splits = 1;
    if (g.epi.kind == GemmEpi::kNone && tiles < sms && g.kchunks >= 16)
        splits = std::min(int(ceil_div(2 * sms, tiles)), g.kchunks / 4);
    g.chunks_per_split = int(ceil_div(g.kchunks, splits));
    splits = int(ceil_div(g.kchunks, g.chunks_per_split));
    g.mode = splits > 1 ? 2 : (accumulate ? 1 : 0);
    if (splits > 1 && !accumulate)
        STB_CUDA(cudaMemset2DAsync(g.C, sizeof(float) * size_t(g.ldc), 0, sizeof(float) * size_t(g.N), size_t(g.M),
                                   st));  // (columns past N are not C's)
    g.err = reinterpret_cast<unsigned long long*>(ctx.flags_d + 8);
    auto kernel = tn ? gemm_bf16_kernel<true> : gemm_bf16_kernel<false>;
    ensure_smem_limit(reinterpret_cast<const void*>(kernel), kGSmem);
    kernel<<<dim3(unsigned(ntiles), unsigned(mtiles), unsigned(splits)), kGThreads, kGSmem, st>>>(g);
    STB_CUDA(cudaGetLastError());
}

}  // namespace

Packed pack_matrix(const PackSrc& s, int rows, int cols, uint8_t* op, cudaStream_t st) {
    if (cols % kGT || !vec_ok(s, cols)) fail(ST_EINVAL, "seqtree_b200: pack_matrix takes aligned rows of 128 columns");
    const int tiles = int(ceil_div(rows, kGT));
    switch (s.kind) {
        case PackSrc::kConv: launch_matrix<PackSrc::kConv>(s, rows, cols, tiles, op, st); break;
        case PackSrc::kRelu: launch_matrix<PackSrc::kRelu>(s, rows, cols, tiles, op, st); break;
        default: launch_matrix<PackSrc::kPlain>(s, rows, cols, tiles, op, st);
    }
    STB_CUDA(cudaGetLastError());
    note_launch(nullptr);
    return Packed{op, rows, cols};
}

void pack_weights(const WeightSrc* w, int n, uint8_t* op, Packed* out, cudaStream_t st) {
    WeightArgs a{};
    if (n < 1 || n > kMaxWeights) fail(ST_EINVAL, "seqtree_b200: pack_weights takes 1 to 10 operands");
    for (int i = 0; i < n; ++i) {
        if (w[i].rows % kGT || w[i].cols % kGK) fail(ST_EINVAL, "seqtree_b200: pack_weights takes whole blocks");
        a.w[i] = w[i];
        a.unit0[i + 1] = a.unit0[i] + int64_t(w[i].rows) * w[i].cols / 8;
        out[i] = Packed{op + a.unit0[i] * 16, w[i].rows, w[i].cols};
    }
    a.op = op;
    pack_weights_kernel<<<unsigned(ceil_div(a.unit0[n], 256)), 256, 0, st>>>(a, n);
    STB_CUDA(cudaGetLastError());
    note_launch(nullptr);
}

void gemm_packed(const Packed& A, const Packed& B, float* C, int ldc, bool accumulate, const GemmEpi& epi,
                 cudaStream_t st, int sms) {
    GemmBf16Args g{};
    g.a = A.op;
    g.b = B.op;
    g.kchunks = A.cols / kGK;
    g.C = C;
    g.ldc = ldc;
    g.M = A.rows;
    g.N = B.rows;
    g.epi = epi;
    run_gemm(g, false, accumulate, st, sms);
    note_launch("gemm_bf16_kernel", 1);
}

void gemm_packed_tn(const Packed& A, const Packed& B, float* C, int ldc, cudaStream_t st, int sms) {
    GemmBf16Args g{};
    g.a = A.op;
    g.b = B.op;
    g.kchunks = 2 * int(ceil_div(A.rows, kGT));  // (rows past the last are packed as zeros)
    g.acols = A.cols / kGK;
    g.bcols = B.cols / kGK;
    g.C = C;
    g.ldc = ldc;
    g.M = A.cols;
    g.N = B.cols;
    run_gemm(g, true, true, st, sms);
    note_launch("gemm_bf16_kernel", 1);
}

// C (=, +=) op(A) op(B) in bf16 with fp32 accumulation.  op(A) is [M x K] (A^T when ta, A being
// [K x M]), op(B) is [K x N] (B^T when tb, B being [N x K]); row-major with leading dimensions.
void gemm_bf16(bool ta, bool tb, int M, int N, int K, const float* A, int lda, const float* B, int ldb,
               float* C, int ldc, bool accumulate, cudaStream_t st, int sms) {
    if (M <= 0 || N <= 0) return;
    if (K <= 0) {
        if (!accumulate)
            STB_CUDA(cudaMemset2DAsync(C, sizeof(float) * size_t(ldc), 0, sizeof(float) * size_t(N),
                                       size_t(M), st));
        return;
    }
    Context& ctx = context();
    ScratchTurn turn(ctx, st);
    PackSrc a{}, b{};
    a.x = A;
    a.ld = lda;
    b.x = B;
    b.ld = ldb;
    GemmBf16Args g{};
    // op(A)[i][k] = ta ? A[k][i] : A[i][k];  op(B)^T[n][k] = tb ? B[n][k] : B[k][n]
    StreamScratch own_a, own_b;
    g.a = pack(a, ta, M, K, turn.as<uint8_t>(ctx.gemm_a, pack_bytes(M, K), own_a), st);
    g.b = pack(b, !tb, N, K, turn.as<uint8_t>(ctx.gemm_b, pack_bytes(N, K), own_b), st);
    g.kchunks = int(ceil_div(K, kGK));
    g.C = C;
    g.ldc = ldc;
    g.M = M;
    g.N = N;
    run_gemm(g, false, accumulate, st, sms);
    note_launch("gemm_bf16_kernel", 3);
}

}  // namespace stb
