// Prefill GEMM on tcgen05 / TMEM and the elementwise steps around it (see prefill.cuh; attention: head_attention.cu).
#include "prefill.cuh"
#include "dense.cuh"
#include "latent.cuh"
#include "ops.cuh"
#include "dequant_bf16.cuh"
#include "tcgen05.cuh"

#include <mutex>

namespace gf {

namespace {

constexpr uint32_t kStages = 3;                                         // shared-memory stages of 64 K elements
constexpr uint32_t kAhead = 2;                                          // stages the activation copies run ahead of the dequantisation
constexpr uint32_t kWeightBufs = 3;                                     // K units of packed weights in shared memory (two in flight)
constexpr uint32_t kPairs = kPrefillTile / 16u;                         // column pairs (16 columns) per CTA
constexpr uint32_t kMaxPairRow = 3360u;                                 // Q6_K
constexpr uint32_t kWeightBufBytes = kPairs * kMaxPairRow;
constexpr uint32_t kAStageBytes = kPrefillBlockBytes;                   // 256 rows x 64 K bf16
constexpr uint32_t kAHalfBytes = kPrefillHalf * kPrefillBlockK * 2u;    // the rows of one accumulator
constexpr uint32_t kBStageBytes = kPrefillTile * kPrefillBlockK * 2u;   // 128 columns x 64 K bf16
constexpr uint32_t kOffA = 0u, kOffB = kStages * kAStageBytes, kOffW = kOffB + kStages * kBStageBytes;
constexpr uint32_t kOffBars = kOffW + kWeightBufs * kWeightBufBytes;
constexpr uint32_t kDequantWarps = 16;                                  // warps 0..15 dequantise; warp 16 requests copies and issues the products
constexpr uint32_t kBarCount = 2u * kWeightBufs + 3u * kStages + 1u;    // weights full / free, per stage: activations landed, weights written, stage free; all done
constexpr uint32_t kPrefillSmemBytes = kOffBars + kBarCount * 8u + 16u;
static_assert(kPrefillSmemBytes <= 227u * 1024u - 1024u, "the GEMM's stages do not fit in one SM's shared memory");

constexpr uint32_t kInstruction = mma_instruction(kPrefillHalf, kPrefillTile);
constexpr uint32_t kTmemColumns = 2u * kPrefillTile;                    // one accumulator of kPrefillTile columns per half of the rows

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// C[128, 128-column tile] = A[128, K] x deq(W)^T.  Grid: (tiles over all matrices of the launch, K splits);
// split s handles its share of the K units and writes its own [128][n] partial result.
//
// Warp-specialised, no block-wide barrier in the loop.  Warps 0..15 dequantise: two warps share a column pair
// of the tile, a lane takes one column of one lane slot; for every 64-element K block they wait until the
// stage is free, write their part of the bf16 weight tile and arrive on the stage's "written" barrier.  One
// thread of warp 17 requests the copies (packed weights two K units ahead, activation blocks two stages
// ahead); one thread of warp 16, once a stage's activations have landed and its weights are written, issues
// the four tensor-core products of the stage; their completion frees the stage.  (With one thread doing
// both, its serial waits, copy requests and issues took longer per stage than the dequantisation.)  Every wait is bounded and gives up
// early once any warp has; the CTA always reaches the end, releases its tensor memory and sets the error word.
__global__ void __launch_bounds__(kPrefillThreads, 1) prefill_gemm_kernel(const __grid_constant__ PrefillGemmParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint32_t tmem_slot;
    __shared__ uint32_t abort_flag;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kOffBars);
    uint64_t* weight_full = bars;                                  // [kWeightBufs]  packed weights of a K unit landed (bytes)
    uint64_t* weight_free = bars + kWeightBufs;                    // [kWeightBufs]  all dequantising warps are done with the unit
    uint64_t* a_full = bars + 2 * kWeightBufs;                     // [kStages]      activation block landed (bytes)
    uint64_t* b_full = a_full + kStages;                           // [kStages]      all dequantising warps have written the stage
    uint64_t* stage_free = b_full + kStages;                       // [kStages]      the stage's products have finished
    uint64_t* done_bar = stage_free + kStages;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const volatile uint32_t* abort = &abort_flag;

    uint32_t which = 0;
    if (p.matrices > 1u && blockIdx.x >= p.m[1].first_tile) which = 1;
    if (p.matrices > 2u && blockIdx.x >= p.m[2].first_tile) which = 2;
    const PrefillMatrix& mat = p.m[which];
    const uint32_t tile = blockIdx.x - mat.first_tile, dtype = mat.dtype;
    const uint32_t row_bytes = pair_row_bytes((int)dtype), subs = p.unit_elems / kPrefillBlockK;
    const uint8_t* weights = mat.weight + (size_t)tile * kPairs * p.units * row_bytes;      // pair rows of pair i start i * units * row_bytes further
    // This split's K units and the activation blocks that go with them.
    const uint32_t unit_begin = (uint32_t)((uint64_t)p.units * blockIdx.y / gridDim.y);
    const uint32_t unit_count = (uint32_t)((uint64_t)p.units * (blockIdx.y + 1u) / gridDim.y) - unit_begin;
    const uint32_t steps = unit_count * subs;
    const uint8_t* blocks = p.a + (size_t)unit_begin * subs * kPrefillBlockBytes;

    if (tid == 0) {
        abort_flag = 0u;
        for (uint32_t i = 0; i < kWeightBufs; ++i) { mbar_init(&weight_full[i], 1); mbar_init(&weight_free[i], kDequantWarps); }
        for (uint32_t i = 0; i < kStages; ++i) { mbar_init(&a_full[i], 1); mbar_init(&b_full[i], kDequantWarps); mbar_init(&stage_free[i], 1); }
        mbar_init(done_bar, 1);
        fence_barrier_init();
    }
    if (warp == 0) tmem_alloc(&tmem_slot, kTmemColumns);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = tmem_slot;
    bool ok = true;

    if (warp == kDequantWarps + 1u) {
        // The copy warp: packed weights two K units ahead, activation blocks kAhead stages ahead.
        if (lane == 0) {
            uint32_t requested_units = 0, requested_blocks = 0;
            auto request_weights = [&](uint32_t j) {          // j counts this split's units
                requested_units = j + 1u;
                uint64_t* bar = &weight_full[j % kWeightBufs];
                uint8_t* dst = smem + kOffW + (j % kWeightBufs) * kWeightBufBytes;
                mbar_expect_tx(bar, kPairs * row_bytes);
                for (uint32_t i = 0; i < kPairs; ++i)
                    bulk_load(dst + i * row_bytes, weights + ((size_t)i * p.units + unit_begin + j) * row_bytes, row_bytes, bar);
            };
            auto request_block = [&](uint32_t step) {         // the stage must be free
                requested_blocks = step + 1u;
                const uint32_t stage = step % kStages;
                mbar_expect_tx(&a_full[stage], p.halves * kAHalfBytes);          // rows 0-127 lie in the block's first half
                bulk_load(smem + kOffA + stage * kAStageBytes, blocks + (size_t)step * kPrefillBlockBytes, p.halves * kAHalfBytes, &a_full[stage]);
            };
            for (uint32_t j = 0; j < 2u && j < unit_count; ++j) request_weights(j);
            for (uint32_t step = 0; step < kAhead && step < steps; ++step) request_block(step);
            for (uint32_t step = 0; step < steps && ok; ++step) {
                const uint32_t j = step / subs;
                if (step % subs == 0u && j + 2u < unit_count) {
                    // The buffer two units on held unit j - 1: every dequantising warp must be done with it.
                    if (j >= 1u && !wait_or_abort(&weight_free[(j + 2u) % kWeightBufs], ((j - 1u) / kWeightBufs) & 1u, abort)) { ok = false; break; }
                    request_weights(j + 2u);
                }
                if (step + kAhead < steps) {
                    const uint32_t next = step + kAhead, next_use = next / kStages;
                    if (next_use > 0u && !wait_or_abort(&stage_free[next % kStages], (next_use - 1u) & 1u, abort)) { ok = false; break; }
                    request_block(next);
                }
            }
            // Whether this warp gave up or another did: copies already requested get a bounded chance to
            // land before the shared memory is released (after a clean run every copy has been consumed).
            if (!ok || !wait_or_abort(done_bar, 0u, abort)) {
                ok = false;
                abort_flag = 1u;
                for (uint32_t j = 0; j < unit_count; ++j) {
                    if (j + kWeightBufs < requested_units) continue;
                    if (j >= requested_units) break;
                    mbar_wait(&weight_full[j % kWeightBufs], (j / kWeightBufs) & 1u, 1u << 16);
                }
                for (uint32_t step = 0; step < steps; ++step) {
                    if (step + kStages < requested_blocks) continue;
                    if (step >= requested_blocks) break;
                    mbar_wait(&a_full[step % kStages], (step / kStages) & 1u, 1u << 16);
                }
            }
        }
    } else if (warp == kDequantWarps) {
        // The issuing warp: once a stage's activations have landed and its weights are written, the four
        // tensor-core products of the stage; their completion frees the stage.
        if (lane == 0) {
            for (uint32_t step = 0; step < steps && ok; ++step) {
                const uint32_t stage = step % kStages, use = step / kStages;
                if (!wait_or_abort(&a_full[stage], use & 1u, abort) || !wait_or_abort(&b_full[stage], use & 1u, abort)) { ok = false; break; }
                tc_fence_after_sync();
                const uint32_t a_address = smem_u32(smem + kOffA + stage * kAStageBytes), b_address = smem_u32(smem + kOffB + stage * kBStageBytes);
                for (uint32_t h = 0; h < p.halves; ++h)
#pragma unroll
                    for (uint32_t kk = 0; kk < kPrefillBlockK / 16u; ++kk)
                        mma_bf16(tmem + h * kPrefillTile, operand_descriptor(a_address + h * kAHalfBytes + kk * 256u),
                                 operand_descriptor(b_address + kk * 256u), kInstruction, (step | kk) != 0u ? 1u : 0u);
                mma_commit(&stage_free[stage]);
            }
            if (ok) mma_commit(done_bar);
            else abort_flag = 1u;
        }
    } else {
        // Dequantisation: warp w takes column pair w % 8 of the tile and the column g + 8 * (w / 8) of each lane slot.
        const uint32_t my_pair = warp % kPairs, column_half = warp / kPairs, my_column = my_pair * 16u + (lane >> 2) + 8u * column_half;
        uint32_t step = 0;
        for (uint32_t j = 0; j < unit_count && ok; ++j) {
            if (!wait_or_abort(&weight_full[j % kWeightBufs], (j / kWeightBufs) & 1u, abort)) { ok = false; break; }
            const uint8_t* pair_row = smem + kOffW + (j % kWeightBufs) * kWeightBufBytes + my_pair * row_bytes;
            for (uint32_t sub = 0; sub < subs; ++sub, ++step) {
                const uint32_t stage = step % kStages, use = step / kStages;
                if (use > 0u && !wait_or_abort(&stage_free[stage], (use - 1u) & 1u, abort)) { ok = false; break; }
                uint8_t* b_stage = smem + kOffB + stage * kBStageBytes;
                if (dtype == GF_Q4_K) dequant_q4k(pair_row, sub, lane, column_half, my_column, b_stage);
                else if (dtype == GF_Q6_K) dequant_q6k(pair_row, sub, lane, column_half, my_column, b_stage);
                else dequant_q80(pair_row, sub, lane, column_half, my_column, b_stage);
                fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&b_full[stage]);
            }
            __syncwarp();
            if (lane == 0 && ok) mbar_arrive(&weight_free[j % kWeightBufs]);
        }
        if (!ok && lane == 0) abort_flag = 1u;
        if (ok && !wait_or_abort(done_bar, 0u, abort)) { ok = false; if (lane == 0) abort_flag = 1u; }
    }
    const bool failed = __syncthreads_or(ok ? 0 : 1) != 0;
    if (!failed && warp < kDequantWarps) {
        tc_fence_after_sync();
        // Warp w reads accumulator lanes 32 * (w % 4) .. +31 (its quarter of a half's rows) and a quarter of the columns.
        const uint32_t column0 = (warp >> 2) * (kPrefillTile / 4u);
        for (uint32_t h = 0; h < p.halves; ++h) {
            const uint32_t row = h * kPrefillHalf + (warp & 3u) * 32u + lane;
            float* out = mat.out + (size_t)blockIdx.y * kPrefillRows * mat.n + (size_t)row * mat.n + (size_t)tile * kPrefillTile + column0;
            float v[32];
            tmem_load_32(tmem + (((warp & 3u) * 32u) << 16) + h * kPrefillTile + column0, v);
#pragma unroll
            for (uint32_t i = 0; i < 32u; i += 4u)
                *reinterpret_cast<float4*>(out + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
        }
        tc_fence_before_sync();
    } else if (failed && tid == 0) {
        atomicExch(p.error_flag, 1);
    }
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, kTmemColumns);
}

// ---- elementwise steps.  A thread handles eight consecutive K elements of one row: two 16-byte loads per
// input and one 16-byte store of eight bf16 into the tile-major operand.

__device__ __forceinline__ float block_total(float v, float* scratch) {
    v = warp_sum(v);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    float total = 0.0f;
    for (uint32_t w = 0; w < blockDim.x / 32u; ++w) total += scratch[w];      // the same order in every thread
    __syncthreads();
    return total;
}

__device__ __forceinline__ void load8(const float* p, float (&v)[8]) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void store_a8(uint8_t* a, uint32_t row, uint32_t k, const float (&v)[8]) {
    *reinterpret_cast<uint4*>(a + tile_major_offset(row, k)) =
        make_uint4(bf16_pair(v[0], v[1]), bf16_pair(v[2], v[3]), bf16_pair(v[4], v[5]), bf16_pair(v[6], v[7]));
}

constexpr uint32_t kNormPieces = 8;       // 8-element pieces a thread keeps in registers: rows of up to 16384 values

// One block per row.  x is the sum of `splits` partial results laid [split][128][k] (added in split order).
// Rows beyond `rows` (up to 128) are written as zeros so that the GEMM's unused rows are defined.
__global__ void __launch_bounds__(256) prefill_norm_kernel(const float* __restrict__ x, uint32_t splits, const float* __restrict__ residual,
                                                           const float* __restrict__ gamma0, const float* __restrict__ gamma1,
                                                           float* __restrict__ residual_out, uint8_t* __restrict__ a_out,
                                                           uint32_t rows, uint32_t k, float eps, int mode) {
    __shared__ float scratch[8];
    const uint32_t row = blockIdx.x, pieces = k / 8u;
    if (row >= rows) {
        const float zero[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        if (a_out) for (uint32_t piece = threadIdx.x; piece < pieces; piece += blockDim.x) store_a8(a_out, row, piece * 8u, zero);
        return;
    }
    float v[kNormPieces][8];
    float sum = 0.0f;
#pragma unroll
    for (uint32_t j = 0; j < kNormPieces; ++j) {
        const uint32_t piece = threadIdx.x + j * 256u;
        if (piece >= pieces) break;
        load8(x + (size_t)row * k + piece * 8u, v[j]);
        for (uint32_t split = 1; split < splits; ++split) {
            float more[8];
            load8(x + ((size_t)split * kPrefillRows + row) * k + piece * 8u, more);
#pragma unroll
            for (int i = 0; i < 8; ++i) v[j][i] += more[i];
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) sum = fmaf(v[j][i], v[j][i], sum);
    }
    float inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(block_total(sum, scratch), (float)k), eps)));
    if (mode == 1) {
        float sum2 = 0.0f;
#pragma unroll
        for (uint32_t j = 0; j < kNormPieces; ++j) {
            const uint32_t piece = threadIdx.x + j * 256u;
            if (piece >= pieces) break;
            float r[8], g[8];
            load8(residual + (size_t)row * k + piece * 8u, r);
            load8(gamma0 + piece * 8u, g);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                v[j][i] = __fadd_rn(r[i], __fmul_rn(__fmul_rn(v[j][i], inv), g[i]));
                sum2 = fmaf(v[j][i], v[j][i], sum2);
            }
            *reinterpret_cast<float4*>(residual_out + (size_t)row * k + piece * 8u) = make_float4(v[j][0], v[j][1], v[j][2], v[j][3]);
            *reinterpret_cast<float4*>(residual_out + (size_t)row * k + piece * 8u + 4u) = make_float4(v[j][4], v[j][5], v[j][6], v[j][7]);
        }
        if (!gamma1 || !a_out) return;
        inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(block_total(sum2, scratch), (float)k), eps)));
    }
#pragma unroll
    for (uint32_t j = 0; j < kNormPieces; ++j) {
        const uint32_t piece = threadIdx.x + j * 256u;
        if (piece >= pieces) break;
        float g[8], out[8];
        load8(gamma1 + piece * 8u, g);
#pragma unroll
        for (int i = 0; i < 8; ++i) out[i] = __fmul_rn(__fmul_rn(v[j][i], inv), g[i]);
        store_a8(a_out, row, piece * 8u, out);
    }
}

// Eight values of row `row` starting at element `at`, summed over `splits` partial results laid [split][128][k].
__device__ __forceinline__ void load8_summed(const float* x, uint32_t splits, uint32_t row, uint32_t k, uint32_t at, float (&v)[8]) {
    load8(x + (size_t)row * k + at, v);
    for (uint32_t split = 1; split < splits; ++split) {
        float more[8];
        load8(x + ((size_t)split * kPrefillRows + row) * k + at, more);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] += more[i];
    }
}

// Grid (128 rows, pieces / 256).  gate and up are sums of `splits` partial results.
__global__ void __launch_bounds__(256) prefill_geglu_kernel(const float* __restrict__ gate, const float* __restrict__ up, uint32_t splits,
                                                            uint8_t* __restrict__ a_out, uint32_t rows, uint32_t k) {
    const uint32_t row = blockIdx.x, piece = blockIdx.y * blockDim.x + threadIdx.x;
    if (piece >= k / 8u) return;
    float out[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    if (row < rows) {
        float g[8], u[8];
        load8_summed(gate, splits, row, k, piece * 8u, g);
        load8_summed(up, splits, row, k, piece * 8u, u);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float v = g[i];
            const float inner = __fmul_rn(0.7978845608028654f, __fadd_rn(v, __fmul_rn(__fmul_rn(__fmul_rn(0.044715f, v), v), v)));
            out[i] = __fmul_rn(__fmul_rn(__fmul_rn(0.5f, v), __fadd_rn(1.0f, tanhf(inner))), u[i]);
        }
    }
    store_a8(a_out, row, piece * 8u, out);
}

// In-place sum of K-split partial results, for up to three matrices: x[0][row][:] += x[1..][row][:].
struct ReduceSet { float* x[3]; uint32_t n[3]; uint32_t count, splits; };
__global__ void __launch_bounds__(256) prefill_reduce_kernel(ReduceSet set, uint32_t rows) {
    const uint32_t row = blockIdx.x;
    if (row >= rows) return;
    for (uint32_t m = 0; m < set.count; ++m) {
        const uint32_t n = set.n[m];
        for (uint32_t piece = blockIdx.y * blockDim.x + threadIdx.x; piece < n / 8u; piece += gridDim.y * blockDim.x) {
            float v[8];
            load8_summed(set.x[m], set.splits, row, n, piece * 8u, v);
            float* dst = set.x[m] + (size_t)row * n + piece * 8u;
            *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<float4*>(dst + 4) = make_float4(v[4], v[5], v[6], v[7]);
        }
    }
}

__global__ void __launch_bounds__(256) prefill_pack_kernel(const float* __restrict__ x, uint8_t* __restrict__ a_out, uint32_t rows, uint32_t k) {
    const uint32_t row = blockIdx.x, piece = blockIdx.y * blockDim.x + threadIdx.x;
    if (piece >= k / 8u) return;
    float out[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    if (row < rows) load8(x + (size_t)row * k + piece * 8u, out);
    store_a8(a_out, row, piece * 8u, out);
}

}  // namespace

int launch_prefill_gemm(const PrefillGemmLaunch& launch, int* error_flag, cudaStream_t stream) {
    if (launch.count == 0 || launch.count > 3 || !launch.a || !error_flag) return fail(GF_ERR_INVALID, "prefill GEMM: bad launch");
    PrefillGemmParams p = {};
    uint32_t tiles = 0;
    for (uint32_t i = 0; i < launch.count; ++i) {
        const auto& m = launch.matrices[i];
        if (m.dtype != GF_Q4_K && m.dtype != GF_Q6_K && m.dtype != GF_Q8_0) return fail(GF_ERR_INVALID, "prefill GEMM: unsupported weight dtype %d", m.dtype);
        if (!m.packed || !m.out || m.n == 0 || m.n % kPrefillTile) return fail(GF_ERR_INVALID, "prefill GEMM: N must be a positive multiple of %u", kPrefillTile);
        const uint32_t unit = unit_elements(m.dtype);
        if (p.unit_elems && p.unit_elems != unit) return fail(GF_ERR_INVALID, "prefill GEMM: Q8_0 and K-quant matrices cannot share a launch");
        p.unit_elems = unit;
        p.m[i] = PrefillMatrix{static_cast<const uint8_t*>(m.packed), m.out, (uint32_t)m.n, (uint32_t)m.dtype, tiles};
        tiles += (uint32_t)(m.n / kPrefillTile);
    }
    if (launch.k == 0 || launch.k % p.unit_elems) return fail(GF_ERR_INVALID, "prefill GEMM: K must be a positive multiple of %u", p.unit_elems);
    p.matrices = launch.count;
    p.tiles = tiles;
    p.k = (uint32_t)launch.k;
    p.units = (uint32_t)(launch.k / p.unit_elems);
    if (launch.splits == 0 || launch.splits > p.units) return fail(GF_ERR_INVALID, "prefill GEMM: K splits must be between 1 and the number of K units");
    p.a = static_cast<const uint8_t*>(launch.a);
    p.error_flag = error_flag;
    if (launch.rows == 0 || launch.rows > kPrefillRows) return fail(GF_ERR_INVALID, "prefill GEMM: rows outside [1, %u]", kPrefillRows);
    p.halves = prefill_padded_rows(launch.rows) / kPrefillHalf;
    static std::once_flag once[64];
    int device = 0;
    cudaGetDevice(&device);
    cudaError_t attr_error = cudaSuccess;
    std::call_once(once[device & 63], [&] {
        attr_error = cudaFuncSetAttribute(prefill_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPrefillSmemBytes);
    });
    GF_CUDA(attr_error);
    prefill_gemm_kernel<<<dim3(tiles, launch.splits), kPrefillThreads, kPrefillSmemBytes, stream>>>(p);
    GF_CUDA(cudaGetLastError());
    return GF_OK;
}

uint32_t prefill_gemm_splits(uint64_t n, uint64_t k, int dtype) {
    // CTAs run one per SM, wave after wave: a launch costs ceil(tiles * splits / SMs) waves of 1 / splits of the
    // whole K each.  Take the split with the least time; ties go to fewer splits.
    const uint32_t tiles = (uint32_t)(n / kPrefillTile), units = (uint32_t)(k / unit_elements(dtype)), sms = (uint32_t)sm_count();
    if (tiles >= sms) return 1;         // every SM already has a tile: more CTAs only add partial results
    uint32_t best = 1;
    double best_cost = 1e30;
    for (uint32_t splits = 1; splits <= kPrefillMaxSplits && splits <= units; ++splits) {
        const uint32_t waves = (tiles * splits + sms - 1u) / sms;
        const double cost = (double)waves * ((double)((units + splits - 1u) / splits) + 0.5);      // half a unit of set-up and epilogue per CTA
        if (cost < best_cost - 1e-9) { best_cost = cost; best = splits; }
    }
    return best;
}

int launch_prefill_norm(const float* x, uint32_t splits, const float* residual, const float* gamma0, const float* gamma1,
                        float* residual_out, void* a_out, uint32_t rows, uint32_t k, float eps, int mode, cudaStream_t stream) {
    if (!x || splits == 0 || rows == 0 || rows > kPrefillRows || k == 0 || k % 8u || k > kNormPieces * 256u * 8u
        || (mode == 0 && (!gamma1 || !a_out)) || (mode == 1 && (!residual || !gamma0 || !residual_out)))
        return fail(GF_ERR_INVALID, "prefill norm: bad arguments");
    const uint32_t blocks = a_out ? prefill_padded_rows(rows) : rows;
    prefill_norm_kernel<<<blocks, 256, 0, stream>>>(x, splits, residual, gamma0, gamma1, residual_out, static_cast<uint8_t*>(a_out), rows, k, eps, mode);
    GF_CUDA(cudaGetLastError());
    return GF_OK;
}

int launch_prefill_reduce(float* const* x, const uint64_t* n, uint32_t count, uint32_t splits, uint32_t rows, cudaStream_t stream) {
    if (!x || !n || count == 0 || count > 3 || splits == 0 || rows == 0 || rows > kPrefillRows) return fail(GF_ERR_INVALID, "prefill reduce: bad arguments");
    if (splits == 1) return GF_OK;
    ReduceSet set = {};
    for (uint32_t i = 0; i < count; ++i) { set.x[i] = x[i]; set.n[i] = (uint32_t)n[i]; }
    set.count = count; set.splits = splits;
    prefill_reduce_kernel<<<dim3(rows, 2), 256, 0, stream>>>(set, rows);
    GF_CUDA(cudaGetLastError());
    return GF_OK;
}

int launch_prefill_geglu(const float* gate, const float* up, uint32_t splits, void* a_out, uint32_t rows, uint32_t k, cudaStream_t stream) {
    if (!gate || !up || !a_out || splits == 0 || rows == 0 || rows > kPrefillRows || k % 8u) return fail(GF_ERR_INVALID, "prefill GeGLU: bad arguments");
    prefill_geglu_kernel<<<dim3(prefill_padded_rows(rows), (k / 8u + 255u) / 256u), 256, 0, stream>>>(gate, up, splits, static_cast<uint8_t*>(a_out), rows, k);
    GF_CUDA(cudaGetLastError());
    return GF_OK;
}

bool prefill_attention_supported(const AttentionParams& p) {
    const uint32_t group = p.kv_heads ? p.heads / p.kv_heads : 0u;
    return p.kv_f16 && p.head_dim == 256u && p.kv_heads != 0u && p.heads % p.kv_heads == 0u && (group == 1u || group == 2u || group == 4u);
}

int launch_prefill_attention(const AttentionParams& p, const Operand* result, int* error_flag, cudaStream_t stream) {
    if (!prefill_attention_supported(p) || p.rows == 0) return fail(GF_ERR_INVALID, "prefill attention: unsupported shape");
    HeadAttention a;
    a.q32 = p.q; a.q_scale = p.scale;
    a.k = static_cast<const __half*>(p.private_k); a.v = static_cast<const __half*>(p.private_v);
    a.ring_k = static_cast<const __half*>(p.ring_k); a.ring_v = static_cast<const __half*>(p.ring_v);
    a.ring_mask = p.ring_mask; a.position = p.base_position; a.softcap = p.softcap; a.window = p.window; a.error_flag = error_flag;
    a.rows = p.rows; a.heads = p.heads; a.kv_heads = p.kv_heads; a.dim_pad = a.vdim = a.vdim_pad = 256u;
    if (result) a.result = *result;
    else { a.result.data = p.out; a.result.capacity = p.rows; a.result.k_pad = p.heads * 256u; a.result.f32 = 1u; }
    return launch_head_attention(a, stream);
}

int launch_prefill_pack(const float* x, void* a_out, uint32_t rows, uint32_t k, cudaStream_t stream) {
    if (!x || !a_out || rows == 0 || rows > kPrefillRows || k % 8u) return fail(GF_ERR_INVALID, "prefill pack: bad arguments");
    prefill_pack_kernel<<<dim3(prefill_padded_rows(rows), (k / 8u + 255u) / 256u), 256, 0, stream>>>(x, static_cast<uint8_t*>(a_out), rows, k);
    GF_CUDA(cudaGetLastError());
    return GF_OK;
}

}  // namespace gf

using namespace gf;

extern "C" {

size_t gf_prefill_workspace_bytes(uint64_t k) { return tile_major_bytes(k); }

int gf_prefill_attention(const float* q_dev, const void* ring_k_dev, const void* ring_v_dev, const void* private_k_dev,
                         const void* private_v_dev, float* out_dev, const uint32_t* base_position_dev, uint32_t rows,
                         uint32_t heads, uint32_t kv_heads, uint32_t head_dim, uint32_t ring_rows, uint32_t window, float scale,
                         float softcap, void* stream) {
    if (!q_dev || !ring_k_dev || !ring_v_dev || !private_k_dev || !private_v_dev || !out_dev || !base_position_dev || rows == 0
        || rows > kPrefillRows || ring_rows == 0 || (ring_rows & (ring_rows - 1u)))
        return fail(GF_ERR_INVALID, "gf_prefill_attention: bad arguments (ring rows must be a power of two, rows at most %u)", kPrefillRows);
    const uintptr_t pointers = reinterpret_cast<uintptr_t>(q_dev) | reinterpret_cast<uintptr_t>(ring_k_dev) | reinterpret_cast<uintptr_t>(ring_v_dev)
        | reinterpret_cast<uintptr_t>(private_k_dev) | reinterpret_cast<uintptr_t>(private_v_dev) | reinterpret_cast<uintptr_t>(out_dev);
    if (pointers & 15u) return fail(GF_ERR_INVALID, "gf_prefill_attention: device pointers must be 16-byte aligned");
    AttentionParams p;
    p.q = q_dev; p.ring_k = ring_k_dev; p.ring_v = ring_v_dev; p.private_k = private_k_dev; p.private_v = private_v_dev;
    p.out = out_dev; p.partial_out = nullptr; p.partial_ml = nullptr; p.counters = nullptr;
    p.base_position = base_position_dev;
    p.rows = rows; p.heads = heads; p.kv_heads = kv_heads; p.head_dim = head_dim;
    p.ring_mask = ring_rows - 1u; p.window = window; p.target_parts = 1; p.scale = scale; p.softcap = softcap; p.kv_f16 = 1;
    return launch_prefill_attention(p, nullptr, nullptr, as_stream(stream));
}

int gf_prefill_matmul(int dtype, const void* packed_dev, const float* x_dev, float* y_dev, uint32_t rows, uint64_t k, uint64_t n,
                      void* workspace_dev, void* stream) {
    if (!packed_dev || !x_dev || !y_dev || !workspace_dev || rows == 0 || rows > kPrefillRows)
        return fail(GF_ERR_INVALID, "gf_prefill_matmul: null buffer or rows outside [1, %u]", kPrefillRows);
    if ((reinterpret_cast<uintptr_t>(y_dev) | reinterpret_cast<uintptr_t>(workspace_dev)) & 15u)
        return fail(GF_ERR_INVALID, "gf_prefill_matmul: y and the workspace must be 16-byte aligned");
    static int* flags[64] = {nullptr};
    int device = 0;
    GF_CUDA(cudaGetDevice(&device));
    device &= 63;
    if (!flags[device]) {
        GF_CUDA(cudaMalloc(&flags[device], sizeof(int)));
        GF_CUDA(cudaMemset(flags[device], 0, sizeof(int)));
    }
    cudaStream_t s = as_stream(stream);
    const int status = launch_prefill_pack(x_dev, workspace_dev, rows, (uint32_t)k, s);
    if (status != GF_OK) return status;
    PrefillGemmLaunch launch;
    launch.matrices[0] = {dtype, packed_dev, y_dev, n};
    launch.count = 1;
    launch.k = k;
    launch.a = workspace_dev;
    launch.rows = rows;
    const int launched = launch_prefill_gemm(launch, flags[device], s);
    if (launched != GF_OK) return launched;
    int value = 0;
    GF_CUDA(cudaMemcpyAsync(&value, flags[device], sizeof(int), cudaMemcpyDeviceToHost, s));
    GF_CUDA(cudaStreamSynchronize(s));
    if (value != 0) {
        cudaMemsetAsync(flags[device], 0, sizeof(int), s);
        return fail(GF_ERR_TIMEOUT, "gf_prefill_matmul: a bounded wait gave up");
    }
    return GF_OK;
}

}  // extern "C"
