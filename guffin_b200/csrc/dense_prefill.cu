// Products over a chunk of prompt rows and the elementwise steps between them (see dense.cuh).
#include "dense.cuh"
#include "tcgen05.cuh"

#include <algorithm>
#include <mutex>

namespace gf {

namespace {

// ------------------------------------------------------------------ outputs

// Column n of the result of product `index` for output row `row`.
__device__ __forceinline__ void chunk_store(const ChunkProblem& p, uint32_t index, uint32_t row, uint32_t n, float v) {
    if (p.output == kChunkF32) {
        if (p.row_scale) {
            const float s = p.row_scale[(size_t)row * p.row_scale_ld];
            v *= p.row_scale_sigmoid ? sigmoid(s) : s;
        }
        p.out[(size_t)row * p.out_ld + n] = v;
    } else if (p.output == kChunkLatentQuery) {
        const size_t at = ((size_t)row * p.heads + index) * p.out_ld + n;
        if (p.query_f16) reinterpret_cast<__half*>(p.out)[at] = __float2half_rn(v * p.scale);
        else p.out[at] = v * p.scale;
    } else if (p.output == kChunkHalfRows) {
        const uint32_t column = (p.segment ? n / p.segment * p.segment_pad + n % p.segment : n) + index * p.column_stride;
        __half* out = reinterpret_cast<__half*>(p.out) + (size_t)row * p.out_ld + column;
        *out = __float2half_rn(v * p.scale);
        if (p.segment && n % p.segment + 1u == p.segment)               // the padding takes part in scores
            for (uint32_t i = 1; i <= p.segment_pad - p.segment; ++i) out[i] = __float2half_rn(0.0f);
    } else {
        const uint32_t column = (p.segment ? n / p.segment * p.segment_pad + n % p.segment : n) + index * p.column_stride;
        store_operand(p.result, row, column, p.output == kChunkSquaredRelu ? squared_relu(v) : v);
    }
}
// Column n of a paired product.
__device__ __forceinline__ float chunk_gate(const ChunkProblem& p, float gate, float up) {
    return p.output == kChunkGeluGate ? gelu_tanh(gate) * up : clamped_gate(gate, up, p.limit);
}
__device__ __forceinline__ void chunk_store_gate(const ChunkProblem& p, uint32_t row, uint32_t n, float gate, float up) {
    const float s = p.row_scale ? p.row_scale[(size_t)row * p.row_scale_ld] : 1.0f;
    store_operand(p.result, row, n, chunk_gate(p, gate * s, up * s));
}

__device__ __forceinline__ uint4 bf16_octet(const float (&v)[8]) {
    uint4 r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r.x) : "f"(v[1]), "f"(v[0]));
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r.y) : "f"(v[3]), "f"(v[2]));
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r.z) : "f"(v[5]), "f"(v[4]));
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r.w) : "f"(v[7]), "f"(v[6]));
    return r;
}
__device__ __forceinline__ uint4 half_octet(const float (&v)[8], float scale) {
    uint4 r;
    uint32_t* w = &r.x;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __half2 h = __floats2half2_rn(v[2 * i] * scale, v[2 * i + 1] * scale);
        w[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
    return r;
}

// Columns n .. n + 7 (n a multiple of eight) of an output row at once where they stay together in the result and start
// on a 16-byte boundary; one by one otherwise.
__device__ __forceinline__ void chunk_store8(const ChunkProblem& p, uint32_t index, uint32_t row, uint32_t n, float (&v)[8]) {
    const bool whole = n + 8u <= p.n && p.segment % 8u == 0u;
    const uint32_t column = (p.segment ? n / p.segment * p.segment_pad + n % p.segment : n) + index * p.column_stride;
    if (whole && p.output == kChunkF32 && p.out_ld % 4u == 0u) {
        float s = 1.0f;
        if (p.row_scale) {
            s = p.row_scale[(size_t)row * p.row_scale_ld];
            if (p.row_scale_sigmoid) s = sigmoid(s);
        }
        float* out = p.out + (size_t)row * p.out_ld + n;
        *reinterpret_cast<float4*>(out) = make_float4(v[0] * s, v[1] * s, v[2] * s, v[3] * s);
        *reinterpret_cast<float4*>(out + 4) = make_float4(v[4] * s, v[5] * s, v[6] * s, v[7] * s);
        return;
    }
    if (whole && column % 8u == 0u && (p.output == kChunkOperand || p.output == kChunkSquaredRelu)) {
        if (p.output == kChunkSquaredRelu)
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = squared_relu(v[i]);
        *reinterpret_cast<uint4*>(static_cast<uint8_t*>(p.result.data) + operand_offset(p.result, row, column)) = bf16_octet(v);
        return;
    }
    if (whole && p.out_ld % 8u == 0u && p.output == kChunkLatentQuery && p.query_f16) {
        *reinterpret_cast<uint4*>(reinterpret_cast<__half*>(p.out) + ((size_t)row * p.heads + index) * p.out_ld + n) = half_octet(v, p.scale);
        return;
    }
    if (whole && p.out_ld % 8u == 0u && column % 8u == 0u && p.output == kChunkHalfRows && p.segment == p.segment_pad) {
        *reinterpret_cast<uint4*>(reinterpret_cast<__half*>(p.out) + (size_t)row * p.out_ld + column) = half_octet(v, p.scale);
        return;
    }
#pragma unroll 1
    for (uint32_t i = 0; i < 8u && n + i < p.n; ++i) chunk_store(p, index, row, n + i, v[i]);
}

// ------------------------------------------------------------------ bf16 products on tcgen05

constexpr uint32_t kWindowMax = 256;                                   // token rows of a tile: the product's N
constexpr uint32_t kPairTile = 2u * kDenseTile;                        // weight columns of a tile: the product's M, half of them a CTA's
constexpr uint32_t kStages = 6;                                        // a stage: a CTA's 128 weight columns, then its half of the window's rows, x 64 K
constexpr uint32_t kStageBytes = kDenseTileBytes + kWindowMax / 2u * 128u;
constexpr uint32_t kEpilogueWarps = 8;
constexpr uint32_t kStagedRows = 32;                                   // token rows that go through shared memory at a time on the way out
constexpr uint32_t kStagedLd = kDenseTile + 4u;                        // floats between them
constexpr uint32_t kChunkThreads = (kEpilogueWarps + 2u) * 32u;        // the copying and the issuing warp behind them
constexpr uint32_t kChunkSmem = kStages * kStageBytes + kStagedRows * kStagedLd * 4u;
static_assert(kChunkSmem + 8u * 1024u <= 227u * 1024u, "stages and staged rows do not fit");

__device__ __forceinline__ void epilogue_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kEpilogueWarps * 32u) : "memory"); }

// What one CTA of a pair has to do for tile `t`.
struct ChunkTile {
    const ChunkProblem* m;
    uint32_t index, tile, row0, live, n_rows;      // n_rows: the product's N
    bool mine;                                     // this CTA's half of the columns exists
    const uint8_t *weight, *rows;
};

// Tiles are numbered problem by problem, a product's windows of token rows next to one another so that they find its
// weights in L2.  A grouped problem (experts; the first of its launch) has as many windows as its groups have rows:
// `windows` holds the number before every group.  Where all indices of a problem read the same rows their 128-column
// tiles form one list, so that a pair is only half used at its end.
__device__ __forceinline__ ChunkTile chunk_tile(const ChunkProduct& p, const uint32_t* windows, uint32_t grouped_tiles, uint32_t t, uint32_t rank) {
    ChunkTile out;
    uint32_t which = 0, pair, window, rows;
    if (t < grouped_tiles) {
        const ChunkProblem& m = p.p[0];
        const uint32_t pairs = (m.tiles + 1u) / 2u, at = t / pairs;
        uint32_t low = 0, high = m.count;          // the group with windows[low] <= at < windows[low + 1]
        while (high - low > 1u) {
            const uint32_t middle = (low + high) / 2u;
            if (windows[middle] <= at) low = middle;
            else high = middle;
        }
        const uint32_t mine = windows[low + 1u] - windows[low], local = t - windows[low] * pairs;
        window = local % mine; pair = local / mine;
        out.index = low;
        rows = m.group_rows[low];
        out.row0 = m.group_start[low] + window * kWindowMax;
        rows -= window * kWindowMax;
        out.live = min(kWindowMax, rows);
    } else {
        t -= grouped_tiles;
        while (which + 1u < p.problems && t >= p.p[which + 1u].first_tile) ++which;
        t -= p.p[which].first_tile;
        const uint32_t per = (p.rows + p.window - 1u) / p.window;
        window = t % per; pair = t / per;
        out.row0 = window * p.window;
        out.live = min(p.window, p.rows - out.row0);
        out.index = 0;
    }
    const ChunkProblem& m = p.p[which];
    out.m = &m;
    if (!m.group_rows) {
        if (m.a_block_stride == 0u) {              // one list of tiles
            const uint32_t last = m.tiles * m.count - 1u, line = 2u * pair + rank;
            out.mine = line <= last;
            out.index = min(line, last) / m.tiles;
            out.tile = min(line, last) % m.tiles;
        } else {
            const uint32_t pairs = (m.tiles + 1u) / 2u;
            out.index = pair / pairs;
            pair %= pairs;
        }
    }
    if (m.group_rows || m.a_block_stride != 0u) {
        const uint32_t line = 2u * pair + rank;
        out.mine = line < m.tiles;
        out.tile = min(line, m.tiles - 1u);
    }
    out.n_rows = (out.live + 31u) & ~31u;
    out.weight = m.weight + out.index * m.weight_stride + (size_t)out.tile * m.k_blocks * kDenseTileBytes;
    out.rows = static_cast<const uint8_t*>(m.a.data) + (size_t)(m.a_block0 + out.index * m.a_block_stride) * m.a.capacity * 128u + (size_t)out.row0 * 128u;
    return out;
}

// Two CTAs (a cluster) share a tile of 256 weight columns (the tensor core's A, a CTA's half each) x a window of up to 256
// token rows (its B, half of them copied by each CTA), so the product's N follows the rows there are (an expert may have
// few) and accumulator lanes are output columns.  Per 64 K and SM that is 32 KB of copies for 512 tensor cycles, where one
// CTA with the whole window copied 48 KB and was held up by what L2 delivers.  One pair per two SMs, tile after tile: the
// accumulators have two sets of 256 columns, so a tile's output runs under the next tile's products.
//
// Bound by the tensor core (512 cycles per 64 K and pair tile) and just above it by L2 (66 bytes per cycle and SM measured
// in 16 KB copies: 490 cycles).  Measured, TFLOP/s, beside the one-CTA form this replaced: 2048 rows x 3840 x 30720: 1437;
// 1024 x 2048 x 16384: 1015 (840); 1024 x 8192 x 2048: 706 (590).  Waits on barriers that the other CTA arrives at must not
// acquire at cluster scope: each such poll costs a cache invalidation (the first case took 2.6 times as long), and the
// copies and products are ordered by the barriers themselves.
//
// Warps 0-7 write outputs, one thread of warp 8 requests copies, one thread of warp 9 issues the products (rank 0) or
// passes on that its CTA's copies have landed (rank 1).  Every wait is bounded; a CTA that gives up raises both CTAs'
// abort words, and both always reach the cluster's barriers.
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kChunkThreads, 1) chunk_product_kernel(const __grid_constant__ ChunkProduct p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint32_t tmem_slot, abort_flag;
    __shared__ uint32_t windows[kMaxExperts + 1u];
    __shared__ __align__(8) uint64_t full[kStages];                     // this CTA's copies landed (bytes)
    __shared__ __align__(8) uint64_t peer_full[kStages];                // rank 0: the other CTA's have
    __shared__ __align__(8) uint64_t free_bar[kStages];                 // the stage's products have finished
    __shared__ __align__(8) uint64_t sums_full[2], sums_free[2];        // a set of accumulators is complete; rank 0: read by both CTAs
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, rank = cluster_rank();
    volatile uint32_t* abort = &abort_flag;

    if (tid == 0) {
        abort_flag = 0u;
        for (uint32_t i = 0; i < kStages; ++i) { mbar_init(&full[i], 1); mbar_init(&peer_full[i], 1); mbar_init(&free_bar[i], 1); }
        for (uint32_t i = 0; i < 2u; ++i) { mbar_init(&sums_full[i], 1); mbar_init(&sums_free[i], 2u * kEpilogueWarps); }
        fence_barrier_init();
    }
    const bool grouped = p.p[0].group_rows != nullptr;
    if (warp == 1u && grouped) {                                        // windows before every group
        uint32_t before = 0;
        for (uint32_t first = 0; first < p.p[0].count; first += 32u) {
            const uint32_t e = first + lane;
            uint32_t sum = e < p.p[0].count ? (p.p[0].group_rows[e] + kWindowMax - 1u) / kWindowMax : 0u;
#pragma unroll
            for (int offset = 1; offset < 32; offset <<= 1) {
                const uint32_t other = __shfl_up_sync(0xffffffffu, sum, offset);
                if (lane >= (uint32_t)offset) sum += other;
            }
            if (e < p.p[0].count) windows[e + 1u] = before + sum;
            before += __shfl_sync(0xffffffffu, sum, 31);
        }
        if (lane == 0) windows[0] = 0u;
    }
    __syncwarp();
    if (warp == 0) tmem_alloc_pair(&tmem_slot, 2u * kWindowMax);
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync();                                                     // the other CTA's barriers are ready too
    tc_fence_after_sync();
    const uint32_t tmem = tmem_slot;
    const uint32_t grouped_tiles = grouped ? windows[p.p[0].count] * ((p.p[0].tiles + 1u) / 2u) : 0u, total = grouped_tiles + p.tiles;
    const uint32_t first = blockIdx.x / 2u, pairs = gridDim.x / 2u;
    bool ok = true;
    auto give_up = [&]() {
        ok = false;
        abort_flag = 1u;
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_address(&abort_flag, rank ^ 1u)), "r"(1u) : "memory");
    };

    // The copying and the issuing warp run their loops with all lanes, and one elected lane issues: the copy and product
    // instructions take their operands from uniform registers, and in a branch of a single thread every one of them costs
    // about 50 cycles more.
    if (warp == kEpilogueWarps) {
        uint32_t stage = 0, parity = 1u, issued = 0;                    // parity: of the phase of free_bar that the next use waits for (the first use passes)
        for (uint32_t t = first; t < total && ok; t += pairs) {
            const ChunkTile tile = chunk_tile(p, windows, grouped_tiles, t, rank);
            // This CTA's half of the window; rows behind the last (in eights) are not copied, nor their sums read.
            const uint32_t half = tile.n_rows / 2u, from = rank * half, present = (tile.live + 7u) & ~7u;
            const uint32_t row_bytes = present > from ? min(half, present - from) * 128u : 0u, steps = tile.m->k_blocks;
            const size_t row_step = (size_t)tile.m->a.capacity * 128u;
            const uint8_t *weight = tile.weight, *rows = tile.rows + (size_t)from * 128u;
            for (uint32_t k = 0; k < steps; ++k) {
                if (!wait_or_abort(&free_bar[stage], parity, abort)) { give_up(); break; }
                if (elect_one()) {
                    uint8_t* at = smem + stage * kStageBytes;
                    mbar_expect_tx(&full[stage], kDenseTileBytes + row_bytes);
                    bulk_load(at, weight, kDenseTileBytes, &full[stage]);
                    if (row_bytes) bulk_load(at + kDenseTileBytes, rows, row_bytes, &full[stage]);
                }
                __syncwarp();
                weight += kDenseTileBytes;
                rows += row_step;
                ++issued;
                if (++stage == kStages) { stage = 0; parity ^= 1u; }
            }
        }
        // Copies requested and not waited for by anybody get a bounded chance to land before the memory is released.
        for (uint32_t i = issued > kStages ? issued - kStages : 0u; i < issued; ++i) mbar_wait(&full[i % kStages], (i / kStages) & 1u, ok ? kMbarWaitLimit : 1u << 16);
    } else if (warp == kEpilogueWarps + 1u) {
        uint32_t stage = 0, parity = 0, count = 0;
        const uint64_t first_a = operand_descriptor(smem_u32(smem)), first_b = operand_descriptor(smem_u32(smem) + kDenseTileBytes);
        for (uint32_t t = first; t < total && ok; t += pairs, ++count) {
            const ChunkTile tile = chunk_tile(p, windows, grouped_tiles, t, rank);
            const uint32_t steps = tile.m->k_blocks;
            if (rank != 0u) {
                for (uint32_t k = 0; k < steps; ++k) {
                    if (!wait_or_abort(&full[stage], parity, abort)) { give_up(); break; }
                    if (elect_one()) mbar_arrive_at(cluster_address(&peer_full[stage], 0u));
                    __syncwarp();
                    if (++stage == kStages) { stage = 0; parity ^= 1u; }
                }
                continue;
            }
            const uint32_t set = count & 1u, instruction = mma_instruction(kPairTile, tile.n_rows), sums = tmem + set * kWindowMax;
            if (count >= 2u && !wait_or_abort(&sums_free[set], (count / 2u - 1u) & 1u, abort)) { give_up(); break; }
            tc_fence_after_sync();
            for (uint32_t k = 0; k < steps; ++k) {
                if (!wait_or_abort(&full[stage], parity, abort) || !wait_or_abort(&peer_full[stage], parity, abort)) { give_up(); break; }
                tc_fence_after_sync();
                if (elect_one()) {
                    const uint64_t a = first_a + stage * (kStageBytes / 16u), b = first_b + stage * (kStageBytes / 16u);
#pragma unroll
                    for (uint32_t kk = 0; kk < kDenseBlockK / 16u; ++kk) mma_bf16_pair(sums, a + kk * 16u, b + kk * 16u, instruction, (k | kk) != 0u ? 1u : 0u);
                    mma_commit_pair(&free_bar[stage]);
                    if (k + 1u == steps) mma_commit_pair(&sums_full[set]);
                }
                __syncwarp();
                if (++stage == kStages) { stage = 0; parity ^= 1u; }
            }
        }
    } else {
        // Output, 32 token rows at a time: the accumulators go through shared memory, so that a thread holds eight
        // neighbouring columns of a row.
        float* staged = reinterpret_cast<float*>(smem + kStages * kStageBytes);      // [kStagedRows][kStagedLd]
        const uint32_t quarter = warp & 3u, lanes = (quarter * 32u) << 16, half = (warp >> 2) * 16u;
        uint32_t count = 0;
        for (uint32_t t = first; t < total; t += pairs, ++count) {
            const ChunkTile tile = chunk_tile(p, windows, grouped_tiles, t, rank);
            const ChunkProblem& m = *tile.m;
            const uint32_t set = count & 1u, sums = tmem + set * kWindowMax + lanes;
            if (warp == 0u && !wait_or_abort(&sums_full[set], (count / 2u) & 1u, abort)) give_up();
            __syncwarp();
            // All warps go on or none (they share barriers below).
            uint32_t any;
            asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                         : "=r"(any) : "r"(ok ? 0u : 1u), "n"(kEpilogueWarps * 32u) : "memory");
            if (any) { ok = false; break; }
            tc_fence_after_sync();
            const bool paired = paired_chunk(m.output);
            for (uint32_t c0 = 0; c0 < tile.live; c0 += kStagedRows) {
                float v[16];
                tmem_load_16(sums + c0 + half, v);
                if (c0 + kStagedRows >= tile.live) {                    // this warp's last read of the set
                    tc_fence_before_sync();
                    if (lane == 0) mbar_arrive_at(cluster_address(&sums_free[set], 0u));
                }
                if (!tile.mine) continue;
#pragma unroll
                for (uint32_t i = 0; i < 16u; ++i) staged[(half + i) * kStagedLd + quarter * 32u + lane] = v[i];
                epilogue_sync();
                const uint32_t octets = paired ? 8u : 16u, work = min(kStagedRows, tile.live - c0) * octets;
#pragma unroll 1
                for (uint32_t i = tid; i < work; i += kEpilogueWarps * 32u) {
                    const uint32_t r = i / octets, octet = i % octets, row = tile.row0 + c0 + r;
                    const float* src = staged + r * kStagedLd + octet * (paired ? 16u : 8u);
                    float o[8];
#pragma unroll
                    for (int j = 0; j < 8; j += 4) *reinterpret_cast<float4*>(o + j) = *reinterpret_cast<const float4*>(src + j);
                    if (!paired) {
                        const uint32_t n = tile.tile * kDenseTile + octet * 8u;
                        if (n < m.n) chunk_store8(m, tile.index, row, n, o);
                        continue;
                    }
                    const uint32_t n = tile.tile * (kDenseTile / 2u) + octet * 8u;
                    if (n >= m.n / 2u) continue;
                    const float s = m.row_scale ? m.row_scale[(size_t)row * m.row_scale_ld] : 1.0f;
#pragma unroll
                    for (int j = 0; j < 8; ++j) o[j] = chunk_gate(m, o[j] * s, src[8 + j] * s);
                    *reinterpret_cast<uint4*>(static_cast<uint8_t*>(m.result.data) + operand_offset(m.result, row, n)) = bf16_octet(o);
                }
                epilogue_sync();
            }
        }
    }
    const bool failed = __syncthreads_or(ok ? 0 : 1) != 0;
    if (failed && tid == 0) atomicExch(p.error_flag, 1);
    __syncwarp();
    tc_fence_before_sync();
    cluster_sync();                                                     // nobody reads the other CTA's shared memory or accumulators any more
    tc_fence_after_sync();
    if (warp == 0) tmem_dealloc_pair(tmem, 2u * kWindowMax);
}

// ------------------------------------------------------------------ f32 products

// 64 rows x 64 columns per CTA, 4 x 4 per thread; a thread's columns are two (gate, up) pairs of a paired matrix.
__global__ void __launch_bounds__(256) chunk_product_f32_kernel(const __grid_constant__ ChunkProduct p) {
    __shared__ float a_tile[32][65], w_tile[32][65];
    const uint32_t tid = threadIdx.x;
    uint32_t which = 0;
    while (which + 1u < p.problems && blockIdx.x >= p.p[which + 1u].first_tile) ++which;
    const ChunkProblem& m = p.p[which];
    const uint32_t index = (blockIdx.x - m.first_tile) / m.tiles, tile = (blockIdx.x - m.first_tile) % m.tiles;
    const uint32_t start = m.group_start ? m.group_start[index] : 0u, rows = m.group_rows ? m.group_rows[index] : p.rows;
    const uint32_t first_row = blockIdx.y * 64u;
    if (first_row >= rows) return;
    const uint32_t live = min(64u, rows - first_row), row0 = start + first_row;
    const uint8_t* weight = m.weight + index * m.weight_stride;
    const float* a = static_cast<const float*>(m.a.data) + (size_t)(m.a_block0 + index * m.a_block_stride) * kDenseBlockK;
    const uint32_t tx = tid & 15u, ty = tid >> 4, column0 = (tx >> 3) * 16u + (tx & 7u);
    const uint32_t columns[4] = {column0, column0 + 8u, column0 + 32u, column0 + 40u};
    float acc[4][4] = {};
    for (uint32_t k0 = 0; k0 < m.k; k0 += 32u) {
        for (uint32_t i = tid; i < 64u * 32u; i += 256u) {
            const uint32_t r = i >> 5, k = i & 31u;
            a_tile[k][r] = r < live && k0 + k < m.k ? a[(size_t)(row0 + r) * m.a.k_pad + k0 + k] : 0.0f;
        }
        {
            const uint32_t n = tid & 63u, piece = tid >> 6;            // 64 columns x four pieces of eight
            const uint4 v = *reinterpret_cast<const uint4*>(weight + dense_offset(m.k_blocks, tile * 64u + n, k0 + piece * 8u));
            const uint32_t words[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (uint32_t j = 0; j < 4u; ++j) {
                w_tile[piece * 8u + 2u * j][n] = __uint_as_float(words[j] << 16);
                w_tile[piece * 8u + 2u * j + 1u][n] = __uint_as_float(words[j] & 0xffff0000u);
            }
        }
        __syncthreads();
#pragma unroll 8
        for (uint32_t k = 0; k < 32u; ++k) {
            float x[4], w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) { x[i] = a_tile[k][ty * 4u + i]; w[i] = w_tile[k][columns[i]]; }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(x[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }
    for (int i = 0; i < 4; ++i) {
        const uint32_t r = ty * 4u + i;
        if (r >= live) continue;
        if (paired_chunk(m.output)) {
            for (int j = 0; j < 4; j += 2) {
                const uint32_t n = tile * 32u + (columns[j] >> 4) * 8u + (columns[j] & 7u);
                if (n < m.n / 2u) chunk_store_gate(m, row0 + r, n, acc[i][j], acc[i][j + 1]);
            }
        } else {
            for (int j = 0; j < 4; ++j)
                if (tile * 64u + columns[j] < m.n) chunk_store(m, index, row0 + r, tile * 64u + columns[j], acc[i][j]);
        }
    }
}

// ------------------------------------------------------------------ norms, routing, cache rows

__device__ __forceinline__ float block_total(float v, float* scratch) {
    v = warp_sum(v);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    float total = 0.0f;
    for (uint32_t w = 0; w < blockDim.x / 32u; ++w) total += scratch[w];
    __syncthreads();
    return total;
}

__global__ void __launch_bounds__(256) chunk_norm_kernel(const ChunkNorm p) {
    extern __shared__ __align__(16) float row_values[];
    __shared__ float scratch[8];
    const uint32_t row = blockIdx.x;
    float* residual = p.residual + (size_t)row * p.width;
    float sum = 0.0f;
    if (p.width % 8u == 0u && !p.slots && !p.result.f32) {             // whole 16-byte pieces
        auto octet = [](float* to, const float* from) {
#pragma unroll
            for (int j = 0; j < 8; j += 4) *reinterpret_cast<float4*>(to + j) = *reinterpret_cast<const float4*>(from + j);
        };
        float v[8], g[8];
        if (p.y) {
            for (uint32_t i = threadIdx.x * 8u; i < p.width; i += blockDim.x * 8u) {
                octet(v, p.y + (size_t)row * p.width + i);
                octet(row_values + i, v);
#pragma unroll
                for (int j = 0; j < 8; ++j) sum = fmaf(v[j], v[j], sum);
            }
            const float inv = 1.0f / sqrtf(block_total(sum, scratch) / (float)p.width + p.eps);
            sum = 0.0f;
            for (uint32_t i = threadIdx.x * 8u; i < p.width; i += blockDim.x * 8u) {
                float x[8];
                octet(v, residual + i);
                octet(x, row_values + i);
                octet(g, p.gain0 + i);
#pragma unroll
                for (int j = 0; j < 8; ++j) { v[j] += x[j] * inv * g[j]; sum = fmaf(v[j], v[j], sum); }
                octet(residual + i, v);
                octet(row_values + i, v);
            }
        } else {
            for (uint32_t i = threadIdx.x * 8u; i < p.width; i += blockDim.x * 8u) {
                octet(v, residual + i);
                octet(row_values + i, v);
#pragma unroll
                for (int j = 0; j < 8; ++j) sum = fmaf(v[j], v[j], sum);
            }
        }
        const float inv = p.gain1 ? 1.0f / sqrtf(block_total(sum, scratch) / (float)p.width + p.eps) : 1.0f;
        for (uint32_t i = threadIdx.x * 8u; i < p.width; i += blockDim.x * 8u) {
            octet(v, row_values + i);
            if (p.gain1) {
                octet(g, p.gain1 + i);
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = v[j] * inv * g[j];
            }
            if (p.result.data) *reinterpret_cast<uint4*>(static_cast<uint8_t*>(p.result.data) + operand_offset(p.result, row, i)) = bf16_octet(v);
            if (p.normed) octet(p.normed + (size_t)row * p.width + i, v);
        }
        return;
    }
    if (p.y) {
        for (uint32_t i = threadIdx.x; i < p.width; i += blockDim.x) {
            float v;
            if (p.slots) {
                v = 0.0f;
                for (uint32_t s = 0; s < p.slots; ++s) v += p.y[(size_t)p.slot_rows[row * p.slots + s] * p.width + i];
                if (p.shared) v += p.shared[(size_t)row * p.width + i];
            } else v = p.y[(size_t)row * p.width + i];
            row_values[i] = v;
            sum = fmaf(v, v, sum);
        }
        const float inv = 1.0f / sqrtf(block_total(sum, scratch) / (float)p.width + p.eps);
        sum = 0.0f;
        for (uint32_t i = threadIdx.x; i < p.width; i += blockDim.x) {
            const float v = residual[i] + row_values[i] * inv * p.gain0[i];
            residual[i] = v;
            row_values[i] = v;
            sum = fmaf(v, v, sum);
        }
    } else {
        for (uint32_t i = threadIdx.x; i < p.width; i += blockDim.x) {
            const float v = residual[i];
            row_values[i] = v;
            sum = fmaf(v, v, sum);
        }
    }
    const float inv = p.gain1 ? 1.0f / sqrtf(block_total(sum, scratch) / (float)p.width + p.eps) : 1.0f;
    for (uint32_t i = threadIdx.x; i < p.width; i += blockDim.x) {
        const float v = p.gain1 ? row_values[i] * inv * p.gain1[i] : row_values[i];
        if (p.result.data) store_operand(p.result, row, i, v);
        if (p.normed) p.normed[(size_t)row * p.width + i] = v;
    }
}

// Block = (row, part): the part by its own root mean square.
__global__ void __launch_bounds__(256) chunk_part_norm_kernel(const float* __restrict__ x, uint32_t x_ld, const float* __restrict__ gate, uint32_t gate_ld, uint32_t part, const float* __restrict__ gain, float eps,
                                                              const Operand result) {
    extern __shared__ __align__(16) float row_values[];
    __shared__ float scratch[8];
    const uint32_t row = blockIdx.x, first = blockIdx.y * part;
    const float *in = x + (size_t)row * x_ld + first, *z = gate + (size_t)row * gate_ld + first;
    float sum = 0.0f;
    for (uint32_t i = threadIdx.x; i < part; i += blockDim.x) {
        const float v = in[i] * silu(z[i]);
        row_values[i] = v;
        sum = fmaf(v, v, sum);
    }
    const float inv = 1.0f / sqrtf(block_total(sum, scratch) / (float)part + eps);
    for (uint32_t i = threadIdx.x; i < part; i += blockDim.x) store_operand(result, row, first + i, row_values[i] * inv * gain[first + i]);
}

// The same for parts of whole 256 values, bf16: block = row, a thread takes eight values at a time.
__global__ void __launch_bounds__(256) chunk_part_norm_octets_kernel(const float* __restrict__ x, uint32_t x_ld, const float* __restrict__ gate, uint32_t gate_ld,
                                                                     uint32_t width, uint32_t part, const float* __restrict__ gain, float eps, const Operand result) {
    extern __shared__ __align__(16) float row_values[];                // [width], then a sum per 256 values
    float* sums = row_values + width;
    const uint32_t row = blockIdx.x;
    for (uint32_t i = threadIdx.x * 8u; i < width; i += blockDim.x * 8u) {
        float sum = 0.0f;
#pragma unroll
        for (int j = 0; j < 8; j += 4) {
            const float4 v = *reinterpret_cast<const float4*>(x + (size_t)row * x_ld + i + j), z = *reinterpret_cast<const float4*>(gate + (size_t)row * gate_ld + i + j);
            const float4 y = make_float4(v.x * silu(z.x), v.y * silu(z.y), v.z * silu(z.z), v.w * silu(z.w));
            *reinterpret_cast<float4*>(row_values + i + j) = y;
            sum = fmaf(y.x, y.x, fmaf(y.y, y.y, fmaf(y.z, y.z, fmaf(y.w, y.w, sum))));
        }
        sum = warp_sum(sum);
        if ((threadIdx.x & 31u) == 0u) sums[i / 256u] = sum;
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x * 8u; i < width; i += blockDim.x * 8u) {
        const uint32_t first = i / part * (part / 256u);
        float sum = 0.0f, v[8];
        for (uint32_t s = 0; s < part / 256u; ++s) sum += sums[first + s];
        const float inv = 1.0f / sqrtf(sum / (float)part + eps);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = row_values[i + j] * inv * gain[i + j];
        *reinterpret_cast<uint4*>(static_cast<uint8_t*>(result.data) + operand_offset(result, row, i)) = bf16_octet(v);
    }
}

// A warp per row chooses its experts.
__global__ void __launch_bounds__(128) chunk_route_kernel(const ChunkRoute p) {
    extern __shared__ float scores[];                                  // [warps][experts]
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, row = blockIdx.x * 4u + warp;
    if (row >= p.rows) return;
    route_row(p.logits + (size_t)row * p.logits_ld, p.experts, p.top, scores + warp * p.experts, [&](uint32_t slot, uint32_t e, float score) {
        if (lane != 0) return;
        p.slot_experts[row * p.top + slot] = e;
        p.slot_scores[row * p.top + slot] = score;
    });
}

// One block: the experts' counts, their starts, and every choice's grouped row.
__global__ void __launch_bounds__(1024) chunk_starts_kernel(const ChunkRoute p) {
    __shared__ uint32_t counts[kMaxExperts], starts[kMaxExperts];
    for (uint32_t e = threadIdx.x; e < p.experts; e += blockDim.x) counts[e] = 0;
    __syncthreads();
    for (uint32_t at = threadIdx.x; at < p.rows * p.top; at += blockDim.x) p.slot_rows[at] = atomicAdd(&counts[p.slot_experts[at]], 1u);
    __syncthreads();
    if (threadIdx.x < 32u) {                                           // prefix sums of the counts, rounded up to eight
        uint32_t before = 0;
        for (uint32_t first = 0; first < p.experts; first += 32u) {
            const uint32_t e = first + threadIdx.x, padded = e < p.experts ? (counts[e] + 7u) & ~7u : 0u;
            uint32_t sum = padded;
#pragma unroll
            for (int offset = 1; offset < 32; offset <<= 1) {
                const uint32_t other = __shfl_up_sync(0xffffffffu, sum, offset);
                if (threadIdx.x >= (uint32_t)offset) sum += other;
            }
            if (e < p.experts) starts[e] = before + sum - padded;
            before += __shfl_sync(0xffffffffu, sum, 31);
        }
    }
    __syncthreads();
    for (uint32_t e = threadIdx.x; e < p.experts; e += blockDim.x) { p.group_start[e] = starts[e]; p.group_rows[e] = counts[e]; }
    for (uint32_t at = threadIdx.x; at < p.rows * p.top; at += blockDim.x) {
        const uint32_t grouped = starts[p.slot_experts[at]] + p.slot_rows[at];
        p.slot_rows[at] = grouped;
        p.row_scale[grouped] = p.slot_scores[at];
    }
}

// Copies a token's normalised row to its grouped rows, 16 bytes at a time.
__global__ void __launch_bounds__(256) chunk_group_kernel(const ChunkRoute p) {
    const uint32_t at = blockIdx.x, row = at / p.top, grouped = p.slot_rows[at];
    if (p.from.f32) {
        const float4* src = reinterpret_cast<const float4*>(static_cast<const float*>(p.from.data) + (size_t)row * p.from.k_pad);
        float4* dst = reinterpret_cast<float4*>(static_cast<float*>(p.to.data) + (size_t)grouped * p.to.k_pad);
        for (uint32_t i = threadIdx.x; i < p.from.k_pad / 4u; i += blockDim.x) dst[i] = src[i];
        return;
    }
    for (uint32_t i = threadIdx.x; i < p.from.k_pad / 8u; i += blockDim.x)
        *reinterpret_cast<uint4*>(static_cast<uint8_t*>(p.to.data) + operand_offset(p.to, grouped, i * 8u)) =
            *reinterpret_cast<const uint4*>(static_cast<const uint8_t*>(p.from.data) + operand_offset(p.from, row, i * 8u));
}

__global__ void __launch_bounds__(256) chunk_operand_kernel(const float* __restrict__ x, uint32_t k, const Operand result) {
    for (uint32_t i = threadIdx.x; i < result.k_pad; i += blockDim.x) store_operand(result, blockIdx.x, i, i < k ? x[(size_t)blockIdx.x * k + i] : 0.0f);
}

__global__ void __launch_bounds__(128) chunk_latents_kernel(const float* __restrict__ raw, uint32_t raw_ld, const float* __restrict__ gain, uint32_t rank,
                                                            float eps, void* cache_rows, uint32_t row_elements, bool f16, uint32_t* status) {
    __shared__ float scratch[8];
    const uint32_t row = blockIdx.x;
    const float* x = raw + (size_t)row * raw_ld;
    float sum = 0.0f;
    for (uint32_t i = threadIdx.x; i < rank; i += blockDim.x) sum = fmaf(x[i], x[i], sum);
    const float inv = 1.0f / sqrtf(block_total(sum, scratch) / (float)rank + eps);
    for (uint32_t i = threadIdx.x; i < row_elements; i += blockDim.x) {
        const float v = i < rank ? x[i] * inv * gain[i] : 0.0f;
        const size_t at = (size_t)row * row_elements + i;
        if (f16) {
            const __half h = __float2half_rn(v);
            if (__hisinf(h) || __hisnan(h)) atomicOr(status, kStatusKvNonFinite);
            static_cast<__half*>(cache_rows)[at] = h;
        } else static_cast<float*>(cache_rows)[at] = v;
    }
}

template <typename Kernel>
int allow_smem(Kernel kernel, std::once_flag* once, uint32_t bytes) {
    int device = 0;
    cudaGetDevice(&device);
    cudaError_t error = cudaSuccess;
    std::call_once(once[device & 63], [&] { error = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes); });
    GF_CUDA(error);
    return GF_OK;
}

}  // namespace

int launch_chunk_product(ChunkProduct p, bool f32, cudaStream_t stream) {
    if (p.problems == 0 || p.problems > 3 || p.rows == 0 || !p.error_flag) return fail(GF_ERR_INVALID, "chunk product: bad launch");
    const uint32_t tile_columns = f32 ? 64u : kDenseTile;
    uint32_t total = 0;
    for (uint32_t i = 0; i < p.problems; ++i) {
        ChunkProblem& m = p.p[i];
        if (!m.weight || !m.a.data || m.n == 0 || m.k == 0 || m.count == 0 || m.a.f32 != (f32 ? 1u : 0u)) return fail(GF_ERR_INVALID, "chunk product: bad problem");
        if (m.group_rows && (!m.group_start || (!f32 && (i != 0u || m.count > kMaxExperts)))) return fail(GF_ERR_INVALID, "chunk product: bad groups");
        m.k_blocks = (m.k + kDenseBlockK - 1u) / kDenseBlockK;
        if ((m.a_block0 + (m.count - 1u) * m.a_block_stride + m.k_blocks) * kDenseBlockK > m.a.k_pad) return fail(GF_ERR_INVALID, "chunk product: the operand is narrower than K");
        if (!m.group_rows && p.rows > m.a.capacity) return fail(GF_ERR_INVALID, "chunk product: more rows than the operand holds");
        m.first_tile = total;
        m.tiles = (m.n + tile_columns - 1u) / tile_columns;
        total += m.tiles * m.count;
    }
    if (f32) {
        p.window = 64u;
        chunk_product_f32_kernel<<<dim3(total, (p.rows + 63u) / 64u), 256, 0, stream>>>(p);
        GF_CUDA(cudaGetLastError());
        return GF_OK;
    }
    // Pairs of 128-column tiles, and the window of rows with the least time: waves of tiles x what a K block of one costs,
    // 2 cycles of the tensor core per row or what its copies take at the 70 bytes per cycle and SM that L2 was seen to
    // deliver, whichever is more, x the largest K (two K blocks more for a tile's start and output).
    auto pairs_of = [](const ChunkProblem& m) {
        return m.group_rows ? 0u : m.a_block_stride == 0u ? (m.tiles * m.count + 1u) / 2u : (m.tiles + 1u) / 2u * m.count;
    };
    const uint32_t clusters = (uint32_t)sm_count() / 2u;
    uint32_t pairs = 0;
    for (uint32_t i = 0; i < p.problems; ++i) pairs += pairs_of(p.p[i]);
    uint64_t best = ~0ull;
    for (uint32_t window = kWindowMax; window >= 32u; window -= 32u) {
        const uint64_t per = (p.rows + window - 1u) / window, waves = (pairs * per + clusters - 1u) / clusters;
        const uint64_t block = std::max<uint64_t>(2u * window, (kDenseTileBytes + 64u * window) / 70u);
        if (waves * block < best) { best = waves * block; p.window = window; }
    }
    const uint32_t per = (p.rows + p.window - 1u) / p.window;
    p.tiles = 0;
    for (uint32_t i = 0; i < p.problems; ++i) {
        p.p[i].first_tile = p.tiles;
        p.tiles += pairs_of(p.p[i]) * per;
    }
    static std::once_flag once[64];
    const int status = allow_smem(chunk_product_kernel, once, kChunkSmem);
    if (status != GF_OK) return status;
    const uint32_t grid = p.p[0].group_rows ? clusters : std::min(clusters, p.tiles);
    chunk_product_kernel<<<2u * grid, kChunkThreads, kChunkSmem, stream>>>(p);
    GF_CUDA(cudaGetLastError());
    return GF_OK;
}

int launch_chunk_norm(const ChunkNorm& p, cudaStream_t stream) {
    if (!p.residual || p.rows == 0 || p.width == 0 || p.width > 48u * 1024u) return fail(GF_ERR_INVALID, "chunk norm: bad arguments");
    static std::once_flag once[64];
    const int status = allow_smem(chunk_norm_kernel, once, 200u * 1024u);
    if (status != GF_OK) return status;
    chunk_norm_kernel<<<p.rows, 256, p.width * 4u, stream>>>(p);
    GF_CUDA(cudaGetLastError());
    return GF_OK;
}

int launch_chunk_part_norm(const float* x, uint32_t x_ld, const float* gate, uint32_t gate_ld, uint32_t width, uint32_t parts, const float* gain, float eps, const Operand& result, uint32_t rows,
                           cudaStream_t stream) {
    if (!x || !gate || !gain || !result.data || rows == 0 || rows > result.capacity || parts == 0 || parts > kMaxNormParts || width % parts || width > result.k_pad
        || width / parts > 48u * 1024u)
        return fail(GF_ERR_INVALID, "chunk part norm: bad arguments");
    const uint32_t part = width / parts;
    static std::once_flag once[2][64];
    int status = allow_smem(chunk_part_norm_kernel, once[0], 200u * 1024u);
    if (status == GF_OK) status = allow_smem(chunk_part_norm_octets_kernel, once[1], 200u * 1024u);
    if (status != GF_OK) return status;
    if (part % 256u == 0u && x_ld % 4u == 0u && gate_ld % 4u == 0u && width <= 40u * 1024u && !result.f32) {
        chunk_part_norm_octets_kernel<<<rows, 256, (width + width / 256u) * 4u, stream>>>(x, x_ld, gate, gate_ld, width, part, gain, eps, result);
        GF_CUDA(cudaGetLastError());
        return GF_OK;
    }
    chunk_part_norm_kernel<<<dim3(rows, parts), part >= 256u ? 256u : (part + 31u) / 32u * 32u, part * 4u, stream>>>(x, x_ld, gate, gate_ld, part, gain, eps, result);
    GF_CUDA(cudaGetLastError());
    return GF_OK;
}

int launch_route(const ChunkRoute& p, cudaStream_t stream) {
    if (p.rows == 0 || p.experts == 0 || p.experts > kMaxExperts || p.top == 0 || p.top > p.experts) return fail(GF_ERR_INVALID, "route: bad arguments");
    chunk_route_kernel<<<(p.rows + 3u) / 4u, 128, 4u * p.experts * 4u, stream>>>(p);
    GF_CUDA(cudaGetLastError());
    return GF_OK;
}

int launch_chunk_route(const ChunkRoute& p, cudaStream_t stream) {
    if (grouped_rows(p.rows, p.top, p.experts) > p.to.capacity) return fail(GF_ERR_INVALID, "chunk route: the grouped operand is too small");
    const int status = launch_route(p, stream);
    if (status != GF_OK) return status;
    chunk_starts_kernel<<<1, 1024, 0, stream>>>(p);
    chunk_group_kernel<<<p.rows * p.top, 256, 0, stream>>>(p);
    GF_CUDA(cudaGetLastError());
    return GF_OK;
}

int launch_chunk_operand(const float* x, uint32_t rows, uint32_t k, const Operand& result, cudaStream_t stream) {
    if (!x || !result.data || rows == 0 || rows > result.capacity || k > result.k_pad) return fail(GF_ERR_INVALID, "chunk operand: bad arguments");
    chunk_operand_kernel<<<rows, 256, 0, stream>>>(x, k, result);
    GF_CUDA(cudaGetLastError());
    return GF_OK;
}

int launch_chunk_latents(const float* raw, uint32_t raw_ld, const float* gain, uint32_t rank, float eps, void* cache_rows, uint32_t row_elements,
                         bool f16, uint32_t rows, uint32_t* status, cudaStream_t stream) {
    chunk_latents_kernel<<<rows, 128, 0, stream>>>(raw, raw_ld, gain, rank, eps, cache_rows, row_elements, f16, status);
    GF_CUDA(cudaGetLastError());
    return GF_OK;
}

}  // namespace gf
