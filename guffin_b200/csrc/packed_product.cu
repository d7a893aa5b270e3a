// Products of a prompt chunk of up to 256 rows with packed weights, decoded on the way to the tensor core (see prompt.cuh).
#include "prompt.cuh"
#include "dequant_bf16.cuh"
#include "tcgen05.cuh"

#include <algorithm>
#include <mutex>

namespace gf {

namespace {

constexpr uint32_t kDecodeWarps = 16, kOutputWarps = 8;                 // then two copying warps and the issuing one
constexpr uint32_t kPackedThreads = (kDecodeWarps + kOutputWarps + 3u) * 32u;
constexpr uint32_t kWeightStages = 4;                                   // of 128 K in tensor memory, 64 columns each
constexpr uint32_t kMostStages = 4;                                     // of the rows, 128 K in shared memory
constexpr uint32_t kFixThreads = (kDecodeWarps + kOutputWarps) * 32u;
constexpr uint32_t kMostUnits = 6;                                      // packed K units in flight
constexpr uint32_t kSumColumns = 256;                                   // tensor-memory columns of the sums; the weights' stages lie behind them
constexpr uint32_t kStageRows = 32, kStageLd = 132;                     // rows that go through shared memory at a time on the way out
constexpr uint32_t kPieceWaitLimit = 1u << 20;                          // polls for the pieces of other CTAs
constexpr uint32_t kPackedSmem = 224u * 1024u;

__device__ __forceinline__ void arrive(uint64_t* bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory"); }
__device__ __forceinline__ void output_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kOutputWarps * 32u) : "memory"); }
// A from tensor memory: 128 lanes x 8 columns of bf16 pairs.
__device__ __forceinline__ void mma_bf16_from_tmem(uint32_t tmem_d, uint32_t tmem_a, uint64_t b_desc, uint32_t instruction, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(b_desc), "r"(instruction), "r"(accumulate) : "memory");
}
// Sixteen lanes x 32 columns: registers 4c .. 4c + 3 are columns 8c + 2t, 8c + 2t + 1 of row g and of row g + 8 (lane 4g + t).
__device__ __forceinline__ void tmem_store_block(uint32_t address, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(address), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
          "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}

// ---- decoding to bf16 pairs: the reference's values, rounded once to bf16.
//
// A code byte q becomes the float 128 + q by one byte permute into the top of the mantissa (0x43000000 | q << 16, q < 128), and
// scale * (128 + q) + (least - 128 scale) in one multiply-add is scale * q + least up to 2^-16 of the scale: a five-hundredth
// of what the rounding to bf16 leaves of a code's value.
__device__ __forceinline__ pf2 pf2_fma(pf2 a, pf2 b, pf2 c) { pf2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ pf2 raw_pair(uint32_t word, uint32_t i) {          // bytes i, i + 1 of `word` (each below 128) plus 128
    pf2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(__byte_perm(word, 0x43000000u, 0x7044u | (i << 8))), "r"(__byte_perm(word, 0x43000000u, 0x7044u | ((i + 1u) << 8))));
    return r;
}
__device__ __forceinline__ void decode_four(uint32_t codes, pf2 scale, pf2 offset, uint32_t& r01, uint32_t& r23) {
    r01 = pf2_bf16(pf2_fma(scale, raw_pair(codes, 0u), offset));
    r23 = pf2_bf16(pf2_fma(scale, raw_pair(codes, 2u), offset));
}
__device__ __forceinline__ float byte_float(uint32_t word, uint32_t i) {      // byte i as a float, exactly
    return __fsub_rn(__uint_as_float(__byte_perm(word, 0x4B000000u, 0x7440u | i)), 8388608.0f);
}
__device__ __forceinline__ pf2 twice(float v) { return pf2_make(v, v); }

}  // namespace

// The K units of all tiles form one list, cut evenly over the CTAs: unit u belongs to CTA share_owner(u).
static __device__ __forceinline__ uint32_t share_begin(uint32_t units, uint32_t ctas, uint32_t cta) { return (uint32_t)((uint64_t)units * cta / ctas); }
static __device__ __forceinline__ uint32_t share_owner(uint32_t units, uint32_t ctas, uint32_t unit) { return (uint32_t)(((uint64_t)(unit + 1u) * ctas - 1u) / units); }

// A CTA takes tiles of 128 weight columns (the tensor core's M) x all rows of the chunk (its N) over a range of K.  Sixteen
// warps decode a K unit's pair rows straight into tensor memory as the A operand, so that decoded weights pass neither through
// HBM nor through shared memory; one warp requests the copies (packed units, 64-K blocks of rows) and one issues the
// products; eight write outputs under the next tile's products.
//
// The (tile, K unit) pairs of a launch are cut evenly over one CTA per SM, so no shape leaves SMs idle.  A tile cut between
// CTAs is parked in pieces in `partial`; at their ends its CTAs each add a share of its rows and write the result.
// Every wait is bounded; a CTA that gives up walks its loops to the end without waiting or issuing.
//
// 128 K at a time: with 64 the issuing warp, which shares its scheduler with six others, took 760 cycles a block of its own
// and bounded everything (3584 x 14336 gate and up, 256 rows: 92 us; now 74, of which products 49, parking and adding pieces
// 16).  Bound at 256 rows by the tensor core (1024 of 2100 cycles per step) and by waiting for the one set of sums to be
// read; for short chunks by the decoding warps (1730 cycles per K unit).  One layer's products of the 9B plan, 192 rows: 165
// us; decoding to HBM and multiplying from there 262, prefill.cu's kernel 270.  191 rows into that plan 14.0 -> 10.5 ms with
// the pass behind them, 65 rows 11.5 -> 9.0; into the 12B plan 16.8 -> 12.7 and 13.7 -> 10.9.
__global__ void __launch_bounds__(kPackedThreads, 1) packed_product_kernel(const __grid_constant__ PackedProduct p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t unit_full[kMostUnits], unit_free[kMostUnits];
    __shared__ __align__(8) uint64_t rows_full[kMostStages], rows_free[kMostStages], weights_full[kWeightStages], weights_free[kWeightStages];
    __shared__ __align__(8) uint64_t sums_full, sums_free;
    __shared__ uint32_t tmem_slot, abort_flag;
    volatile uint32_t* abort = &abort_flag;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    if (tid == 0) {
        abort_flag = 0u;
        for (uint32_t i = 0; i < kMostUnits; ++i) { mbar_init(&unit_full[i], 1); mbar_init(&unit_free[i], kDecodeWarps / 2u); }
        for (uint32_t i = 0; i < kMostStages; ++i) { mbar_init(&rows_full[i], 1); mbar_init(&rows_free[i], 1); }
        for (uint32_t i = 0; i < kWeightStages; ++i) { mbar_init(&weights_full[i], kDecodeWarps / 2u); mbar_init(&weights_free[i], 1); }
        mbar_init(&sums_full, 1);
        mbar_init(&sums_free, kOutputWarps);
        fence_barrier_init();
    }
    if (warp == 0) tmem_alloc(&tmem_slot, 512);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = tmem_slot;
    const uint32_t total = p.tiles * p.units, begin = share_begin(total, gridDim.x, blockIdx.x), end = share_begin(total, gridDim.x, blockIdx.x + 1u);
    const uint32_t steps = p.unit_elems / 128u, stage_bytes = p.n_rows * 256u, unit_bytes = 8u * p.row_bytes;
    uint8_t* units_smem = smem + p.stages * stage_bytes;
    float* staged = reinterpret_cast<float*>(units_smem + p.unit_slots * unit_bytes);
    bool ok = true;
    auto wait = [&](uint64_t* bar, uint32_t parity) {
        if (!ok) return;
        ok = __all_sync(0xffffffffu, mbar_try_wait(bar, parity) || wait_or_abort(bar, parity, abort));
        if (!ok) *abort = 1u;
    };
    auto matrix_of = [&](uint32_t tile) -> uint32_t {
        uint32_t m = 0;
        if (p.paired) return 0u;
        if (p.matrices > 1u && tile >= p.m[1].first_tile) m = 1;
        if (p.matrices > 2u && tile >= p.m[2].first_tile) m = 2;
        return m;
    };

    const uint32_t octets = p.paired ? 8u : 16u;
    auto store = [&](uint32_t tile, uint32_t row, uint32_t octet, float (&o)[8], const float (&up)[8]) {
        if (p.paired) {
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] = gelu_tanh(o[j]) * up[j];
            *reinterpret_cast<uint4*>(static_cast<uint8_t*>(p.result.data) + operand_offset(p.result, row, tile * 64u + octet * 8u)) =
                make_uint4(bf16_pair(o[0], o[1]), bf16_pair(o[2], o[3]), bf16_pair(o[4], o[5]), bf16_pair(o[6], o[7]));
            return;
        }
        const PackedProduct::Matrix& m = p.m[matrix_of(tile)];
        float* out = m.out + (size_t)row * m.n + (tile - m.first_tile) * 128u + octet * 8u;
        *reinterpret_cast<float4*>(out) = make_float4(o[0], o[1], o[2], o[3]);
        *reinterpret_cast<float4*>(out + 4) = make_float4(o[4], o[5], o[6], o[7]);
    };

    if (warp == kDecodeWarps + kOutputWarps) {
        // ---- packed units: a lane per column pair
        uint32_t slot = 0, parity = 1u, requested = 0, tile = begin / p.units, unit = begin % p.units, row = 0, bytes = 0;
        const uint8_t* src = nullptr;
        bool fresh = true;
        for (uint32_t u = begin; u < end; ++u) {
            if (fresh) {
                const uint32_t which = matrix_of(tile), i = lane & 7u;
                const PackedProduct::Matrix& m = p.m[p.paired ? i >> 2 : which];
                const uint32_t pair = p.paired ? tile * 4u + (i & 3u) : (tile - m.first_tile) * 8u + i;
                row = pair_row_bytes((int)m.dtype);
                bytes = p.paired ? 4u * (pair_row_bytes((int)p.m[0].dtype) + pair_row_bytes((int)p.m[1].dtype)) : 8u * row;
                src = m.packed + ((size_t)pair * p.units + unit) * row;
                fresh = false;
            }
            wait(&unit_free[slot], parity);
            if (ok) {
                if (lane == 0) mbar_expect_tx(&unit_full[slot], bytes);
                __syncwarp();
                if (lane < 8u) bulk_load(units_smem + slot * unit_bytes + lane * p.row_bytes, src, row, &unit_full[slot]);
                __syncwarp();
                ++requested;
            }
            src += row;
            if (++unit == p.units) { unit = 0; ++tile; fresh = true; }
            if (++slot == p.unit_slots) { slot = 0; parity ^= 1u; }
        }
        for (uint32_t i = requested > p.unit_slots ? requested - p.unit_slots : 0u; i < requested; ++i)
            mbar_wait(&unit_full[i % p.unit_slots], (i / p.unit_slots) & 1u, ok ? kMbarWaitLimit : 1u << 16);
    } else if (warp == kDecodeWarps + kOutputWarps + 1u) {
        // ---- the rows, two blocks of 64 K at a time
        const size_t row_step = (size_t)p.a.capacity * 128u;
        const uint32_t present = ((p.rows + 7u) & ~7u) * 128u, blocks = (end - begin) * steps, per_tile = p.units * steps;
        const uint8_t* const start = static_cast<const uint8_t*>(p.a.data);
        uint32_t stage = 0, parity = 1u, requested = 0, at = begin % p.units * steps;
        const uint8_t* src = start + 2u * at * row_step;
        for (uint32_t i = 0; i < blocks; ++i) {
            wait(&rows_free[stage], parity);
            if (ok && elect_one()) {
                mbar_expect_tx(&rows_full[stage], 2u * present);
                bulk_load(smem + stage * stage_bytes, src, present, &rows_full[stage]);
                bulk_load(smem + stage * stage_bytes + stage_bytes / 2u, src + row_step, present, &rows_full[stage]);
            }
            __syncwarp();
            if (ok) ++requested;
            src += 2u * row_step;
            if (++at == per_tile) { at = 0; src = start; }
            if (++stage == p.stages) { stage = 0; parity ^= 1u; }
        }
        for (uint32_t i = requested > p.stages ? requested - p.stages : 0u; i < requested; ++i)
            mbar_wait(&rows_full[i % p.stages], (i / p.stages) & 1u, ok ? kMbarWaitLimit : 1u << 16);
    } else if (warp == kDecodeWarps + kOutputWarps + 2u) {
        // ---- products
        const uint32_t instruction = mma_instruction(128, p.n_rows), blocks = (end - begin) * steps, per_tile = p.units * steps;
        const uint64_t rows_at = operand_descriptor(smem_u32(smem));
        uint32_t stage = 0, parity = 0, weights = 0, weights_parity = 0, at = begin % p.units * steps, pieces = 0;
        bool opens = true;
        for (uint32_t i = 0; i < blocks; ++i) {
            if (opens) {
                if (pieces) wait(&sums_free, (pieces - 1u) & 1u);
                ++pieces;
            }
            const bool closes = at + 1u == per_tile || i + 1u == blocks;
            wait(&rows_full[stage], parity);
            wait(&weights_full[weights], weights_parity);
            tc_fence_after_sync();
            if (ok && elect_one()) {
                const uint64_t b = rows_at + stage * (stage_bytes / 16u);
                const uint32_t a = tmem + kSumColumns + weights * 64u;
                mma_bf16_from_tmem(tmem, a, b, instruction, opens ? 0u : 1u);
#pragma unroll
                for (uint32_t kk = 1; kk < 8u; ++kk) mma_bf16_from_tmem(tmem, a + kk * 8u, b + (kk >> 2) * (stage_bytes / 32u) + (kk & 3u) * 16u, instruction, 1u);
                mma_commit(&rows_free[stage]);
                mma_commit(&weights_free[weights]);
                if (closes) mma_commit(&sums_full);
            }
            __syncwarp();
            opens = closes;
            at = at + 1u == per_tile ? 0u : at + 1u;
            if (++stage == p.stages) { stage = 0; parity ^= 1u; }
            if (++weights == kWeightStages) { weights = 0; weights_parity ^= 1u; }
        }
        // The last products' arrivals have landed before the shared memory is given back.
        for (uint32_t i = blocks > p.stages ? blocks - p.stages : 0u; i < blocks; ++i) wait(&rows_free[i % p.stages], (i / p.stages) & 1u);
        for (uint32_t i = blocks > kWeightStages ? blocks - kWeightStages : 0u; i < blocks; ++i) wait(&weights_free[i % kWeightStages], (i / kWeightStages) & 1u);
    } else if (warp < kDecodeWarps) {
        // ---- decode: pair `pair` of the tile's eight, every other K unit
        const uint32_t pair = (warp & 3u) * 2u + ((warp >> 2) & 1u), g = lane >> 2;
        const uint32_t lanes = tmem + ((pair * 16u) << 16) + kSumColumns;
        uint32_t r[16];
        for (uint32_t u = begin + (warp >> 3); u < end; u += 2u) {
            const uint32_t at = u - begin, slot = at % p.unit_slots, dtype = p.m[p.paired ? pair >> 2 : matrix_of(u / p.units)].dtype;
            uint32_t block = at * steps;
            wait(&unit_full[slot], (at / p.unit_slots) & 1u);
            const uint8_t* row = units_smem + slot * unit_bytes + pair * p.row_bytes;
            auto put = [&](uint32_t second) {                           // a block of 64 K; two make a stage
                const uint32_t stage = block % kWeightStages;
                if (!second) {
                    wait(&weights_free[stage], (block / kWeightStages & 1u) ^ 1u);
                    tc_fence_after_sync();
                }
                tmem_store_block(lanes + stage * 64u + second * 32u, r);
                if (!second) return;
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) arrive(&weights_full[stage]);
                ++block;
            };
            if (dtype == (uint32_t)GF_Q4_K) {
                const uint4 ha = *reinterpret_cast<const uint4*>(row + 2048u + g * 16u), hb = *reinterpret_cast<const uint4*>(row + 2176u + g * 16u);
                uint32_t scales[2] = {ha.y & 0x3f3f3f3fu, hb.y & 0x3f3f3f3fu}, minima[2] = {ha.z & 0x3f3f3f3fu, hb.z & 0x3f3f3f3fu};
                const float d[2] = {half_bits(ha.x & 0xffffu), half_bits(hb.x & 0xffffu)}, dmin[2] = {half_bits(ha.x >> 16), half_bits(hb.x >> 16)};
#pragma unroll 1
                for (uint32_t half = 0; half < 2u; ++half) {
#pragma unroll
                    for (uint32_t s = 0; s < 2u; ++s) {
                        const uint4 w = *reinterpret_cast<const uint4*>(row + (2u * half + s) * 512u + lane * 16u);
#pragma unroll
                        for (uint32_t col = 0; col < 2u; ++col)
#pragma unroll
                            for (uint32_t nib = 0; nib < 2u; ++nib) {
                                const float ds = __fmul_rn(d[col], byte_float(scales[col], 2u * s + nib)), dm = __fmul_rn(dmin[col], byte_float(minima[col], 2u * s + nib));
                                const pf2 scale = twice(ds), offset = twice(-fmaf(128.0f, ds, dm));
                                decode_four(((col ? w.z : w.x) >> (4u * nib)) & 0x0f0f0f0fu, scale, offset, r[8u * nib + 2u * col], r[8u * nib + 2u * col + 1u]);
                                decode_four(((col ? w.w : w.y) >> (4u * nib)) & 0x0f0f0f0fu, scale, offset, r[8u * nib + 4u + 2u * col], r[8u * nib + 4u + 2u * col + 1u]);
                            }
                        put(s);
                    }
                    scales[0] = (ha.w & 0x0f0f0f0fu) | ((ha.y >> 2) & 0x30303030u); minima[0] = ((ha.w >> 4) & 0x0f0f0f0fu) | ((ha.z >> 2) & 0x30303030u);
                    scales[1] = (hb.w & 0x0f0f0f0fu) | ((hb.y >> 2) & 0x30303030u); minima[1] = ((hb.w >> 4) & 0x0f0f0f0fu) | ((hb.z >> 2) & 0x30303030u);
                }
            } else if (dtype == (uint32_t)GF_Q6_K) {
                const float d[2] = {half_bits(*reinterpret_cast<const unsigned short*>(row + 3328u + g * 2u)), half_bits(*reinterpret_cast<const unsigned short*>(row + 3344u + g * 2u))};
#pragma unroll 1
                for (uint32_t half = 0; half < 2u; ++half) {
                    const uint4 qa = *reinterpret_cast<const uint4*>(row + half * 1536u + lane * 16u), qb = *reinterpret_cast<const uint4*>(row + half * 1536u + 512u + lane * 16u);
                    const uint4 qh = *reinterpret_cast<const uint4*>(row + half * 1536u + 1024u + lane * 16u);
#pragma unroll
                    for (uint32_t upper = 0; upper < 2u; ++upper) {
                        const uint32_t words[2] = {*reinterpret_cast<const uint32_t*>(row + 3072u + g * 16u + 8u * half + 4u * upper) ^ 0x80808080u,
                                                   *reinterpret_cast<const uint32_t*>(row + 3200u + g * 16u + 8u * half + 4u * upper) ^ 0x80808080u};
#pragma unroll
                        for (uint32_t col = 0; col < 2u; ++col)
#pragma unroll
                            for (uint32_t s = 0; s < 2u; ++s) {
                                const uint32_t even = col ? (s ? qb.z : qb.x) : (s ? qa.z : qa.x), odd = col ? (s ? qb.w : qb.y) : (s ? qa.w : qa.y);
                                const uint32_t high = col ? (s ? qh.w : qh.z) : (s ? qh.y : qh.x);
#pragma unroll
                                for (uint32_t qq = 0; qq < 2u; ++qq) {
                                    const float ds = __fmul_rn(d[col], byte_float(words[col], 2u * qq + s) - 128.0f);
                                    const uint32_t codes = (((qq ? odd : even) >> (4u * upper)) & 0x0f0f0f0fu) | (((high >> (2u * (2u * upper + qq))) & 0x03030303u) << 4);
                                    decode_four(codes, twice(ds), twice(-160.0f * ds), r[(2u * qq + s) * 4u + 2u * col], r[(2u * qq + s) * 4u + 2u * col + 1u]);
                                }
                            }
                        put(upper);
                    }
                }
            } else {
                const uint2 da = *reinterpret_cast<const uint2*>(row + 2048u + g * 8u), db = *reinterpret_cast<const uint2*>(row + 2112u + g * 8u);
                const pf2 neg_bias = pf2_make(-(8388608.0f + 128.0f), -(8388608.0f + 128.0f));
#pragma unroll
                for (uint32_t sub = 0; sub < 2u; ++sub) {
#pragma unroll
                    for (uint32_t bb = 0; bb < 2u; ++bb) {
                        const uint4 w = *reinterpret_cast<const uint4*>(row + (2u * sub + bb) * 512u + lane * 16u);
#pragma unroll
                        for (uint32_t col = 0; col < 2u; ++col) {
                            const uint32_t raw = col ? (sub ? db.y : db.x) : (sub ? da.y : da.x);
                            const pf2 scale = twice(half_bits(bb ? raw >> 16 : raw & 0xffffu));
#pragma unroll
                            for (uint32_t j = 0; j < 2u; ++j) {
                                const uint32_t codes = (col ? (j ? w.w : w.z) : (j ? w.y : w.x)) ^ 0x80808080u;      // int8 + 128
                                r[(2u * bb + j) * 4u + 2u * col] = pf2_bf16(pf2_mul(scale, code_pair(codes, 0u, neg_bias)));
                                r[(2u * bb + j) * 4u + 2u * col + 1u] = pf2_bf16(pf2_mul(scale, code_pair(codes, 2u, neg_bias)));
                            }
                        }
                    }
                    put(sub);
                }
            }
            __syncwarp();
            if (lane == 0) arrive(&unit_free[slot]);
        }
    } else {
        // ---- output, 32 rows at a time
        const uint32_t mine = warp - kDecodeWarps, quarter = mine & 3u, half = (mine >> 2) * 16u, sums = tmem + ((quarter * 32u) << 16);
        const uint32_t thread = tid - kDecodeWarps * 32u;
        uint32_t pieces = 0;
        for (uint32_t u = begin; u < end; ++pieces) {
            const uint32_t tile = u / p.units, tile_begin = tile * p.units, next = min(end, tile_begin + p.units);
            const bool whole = u == tile_begin && next == tile_begin + p.units;
            const size_t piece_floats = (size_t)p.n_rows * 128u;
            float* park = p.partial + (2u * blockIdx.x + (u > tile_begin ? 0u : 1u)) * piece_floats;
            wait(&sums_full, pieces & 1u);
            tc_fence_after_sync();
            for (uint32_t c0 = 0; c0 < p.rows; c0 += kStageRows) {
                float v[16];
                tmem_load_16(sums + c0 + half, v);
                if (c0 + kStageRows >= p.rows) {                        // this warp's last read of the sums
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) arrive(&sums_free);
                }
                if (!whole) {
#pragma unroll
                    for (uint32_t i = 0; i < 16u; ++i) __stcg(&park[(size_t)(c0 + half + i) * 128u + quarter * 32u + lane], v[i]);
                    continue;
                }
#pragma unroll
                for (uint32_t i = 0; i < 16u; ++i) staged[(half + i) * kStageLd + quarter * 32u + lane] = v[i];
                output_sync();
                for (uint32_t i = thread; i < min(kStageRows, p.rows - c0) * octets; i += kOutputWarps * 32u) {
                    const uint32_t row = i / octets, octet = i % octets;
                    const float* src = staged + row * kStageLd + octet * 8u;
                    float o[8], up[8];
#pragma unroll
                    for (int j = 0; j < 8; j += 4) {
                        *reinterpret_cast<float4*>(o + j) = *reinterpret_cast<const float4*>(src + j);
                        if (p.paired) *reinterpret_cast<float4*>(up + j) = *reinterpret_cast<const float4*>(src + 64 + j);
                    }
                    store(tile, c0 + row, octet, o, up);
                }
                output_sync();
            }
            if (!whole) {
                __threadfence();
                output_sync();
                if (thread == 0) atomicAdd(&p.counters[2u * tile], 1u);
            }
            u = next;
        }
    }
    if (warp < kDecodeWarps + kOutputWarps) {
        // Tiles cut between CTAs (the first and the last of this one's): once all pieces are parked, every CTA that has one
        // adds a share of the rows, in the order of K.  All CTAs are resident (a cooperative launch).
        asm volatile("bar.sync 2, %0;" ::"n"(kFixThreads) : "memory");      // nobody polls while its CTA still works
        const uint32_t first_tile = begin / p.units, last_tile = (end - 1u) / p.units;
        for (uint32_t tile = first_tile; tile <= last_tile; tile += max(1u, last_tile - first_tile)) {
            const uint32_t tile_begin = tile * p.units;
            if (begin <= tile_begin && end >= tile_begin + p.units) continue;
            const uint32_t low = share_owner(total, gridDim.x, tile_begin), high = share_owner(total, gridDim.x, tile_begin + p.units - 1u), pieces_of = high - low + 1u;
            if (ok) {
                bool there = false;
                for (uint32_t spin = 0; spin < kPieceWaitLimit && !there; ++spin) {
                    uint32_t count;
                    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(count) : "l"(&p.counters[2u * tile]) : "memory");
                    there = count >= pieces_of;
                    if (*abort != 0u) break;
                    if (!there) __nanosleep(100);
                }
                ok = __all_sync(0xffffffffu, there);
                if (!ok) *abort = 1u;
            }
            const uint32_t from = p.rows * (blockIdx.x - low) / pieces_of, to = p.rows * (blockIdx.x - low + 1u) / pieces_of;
            const size_t piece_floats = (size_t)p.n_rows * 128u;
            // Pieces lie two to a CTA: the one that begins inside a tile, then the one that ends inside a tile.
            const float* head = p.partial + (2u * low + (share_begin(total, gridDim.x, low) > tile_begin ? 0u : 1u)) * piece_floats;
            const float* rest = p.partial + (2u * low + 2u) * piece_floats;
            if (ok)
                for (uint32_t i = from * octets + tid; i < to * octets; i += kFixThreads) {
                    const uint32_t row = i / octets, octet = i % octets;
                    const size_t at = (size_t)row * 128u + octet * 8u;
                    float o[8], up[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) o[j] = up[j] = 0.0f;
                    auto add = [&](float (&to_)[8], const float4& x, const float4& y) {
                        to_[0] += x.x; to_[1] += x.y; to_[2] += x.z; to_[3] += x.w; to_[4] += y.x; to_[5] += y.y; to_[6] += y.z; to_[7] += y.w;
                    };
                    for (uint32_t piece = 0; piece < pieces_of; piece += 4u) {
                        float4 v[4][2];
#pragma unroll
                        for (uint32_t j = 0; j < 4u; ++j)
                            if (piece + j < pieces_of) {
                                const float* src = (piece + j == 0u ? head : rest + (size_t)(piece + j - 1u) * 2u * piece_floats) + at;
                                v[j][0] = __ldcg(reinterpret_cast<const float4*>(src));
                                v[j][1] = __ldcg(reinterpret_cast<const float4*>(src + 4));
                            }
#pragma unroll
                        for (uint32_t j = 0; j < 4u; ++j)
                            if (piece + j < pieces_of) add(o, v[j][0], v[j][1]);
                    }
                    if (p.paired)
                        for (uint32_t piece = 0; piece < pieces_of; ++piece) {
                            const float* src = (piece == 0u ? head : rest + (size_t)(piece - 1u) * 2u * piece_floats) + at + 64u;
                            add(up, __ldcg(reinterpret_cast<const float4*>(src)), __ldcg(reinterpret_cast<const float4*>(src + 4)));
                        }
                    store(tile, row, octet, o, up);
                }
            asm volatile("bar.sync 2, %0;" ::"n"(kFixThreads) : "memory");
            if (tid == 0 && atomicAdd(&p.counters[2u * tile + 1u], 1u) + 1u == pieces_of) {      // the last to leave clears both
                p.counters[2u * tile] = 0u;
                p.counters[2u * tile + 1u] = 0u;
            }
        }
    }
    const bool failed = __syncthreads_or(ok ? 0 : 1) != 0;
    if (failed && tid == 0) atomicExch(p.error_flag, 1);
    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    if (warp == 0) tmem_dealloc(tmem, 512);
}

size_t packed_partial_bytes() { return (size_t)sm_count() * 2u * kPackedRows * 128u * sizeof(float); }

int launch_packed_product(PackedProduct p, cudaStream_t stream) {
    if (p.matrices == 0 || p.matrices > 3u || p.rows == 0 || p.rows > kPackedRows || !p.a.data || p.a.f32 || !p.partial || !p.counters || !p.error_flag
        || (p.paired && (p.matrices != 2u || p.m[0].n != p.m[1].n || !p.result.data)))
        return fail(GF_ERR_INVALID, "packed product: bad launch");
    p.tiles = 0; p.unit_elems = 0; p.row_bytes = 0;
    for (uint32_t i = 0; i < p.matrices; ++i) {
        PackedProduct::Matrix& m = p.m[i];
        const uint32_t unit = unit_elements((int)m.dtype);
        if (!m.packed || m.n == 0 || m.n % 128u || (!p.paired && !m.out) || (p.unit_elems && p.unit_elems != unit)) return fail(GF_ERR_INVALID, "packed product: bad matrix");
        p.unit_elems = unit;
        p.row_bytes = std::max(p.row_bytes, pair_row_bytes((int)m.dtype));
        m.first_tile = p.paired ? 0u : p.tiles;
        p.tiles += m.n / 128u;                               // a pair's tile: 64 columns of each
    }
    if (p.k == 0 || p.k % p.unit_elems) return fail(GF_ERR_INVALID, "packed product: K must be a positive multiple of %u", p.unit_elems);
    p.units = p.k / p.unit_elems;
    p.n_rows = (p.rows + 31u) & ~31u;
    const uint32_t staged = kStageRows * kStageLd * 4u, left = kPackedSmem - staged, unit_bytes = 8u * p.row_bytes;
    // Two packed units at least and as many stages as then fit; what is left goes to more units.
    p.stages = std::min(kMostStages, (left - 2u * unit_bytes) / (p.n_rows * 256u));
    p.unit_slots = std::min(kMostUnits, (left - p.stages * p.n_rows * 256u) / unit_bytes);
    // Cutting tiles evenly over all SMs (a share of at least 512 elements of K) costs parking and adding up the pieces, about
    // 14000 cycles; 128 elements of K cost about 600 + 2 per row.  A tile per CTA where that is no slower: the small matrices
    // of a drafter.
    const uint32_t total = p.tiles * p.units, steps = p.unit_elems / 128u, sms = (uint32_t)sm_count(), cycles = 600u + 2u * p.n_rows;
    uint32_t grid = std::max(1u, std::min(sms, total / (4u / steps)));
    if (p.tiles <= sms && (size_t)p.units * steps * cycles <= (size_t)((total + grid - 1u) / grid) * steps * cycles + 14000u) grid = p.tiles;
    static std::once_flag once[64];
    int device = 0;
    cudaGetDevice(&device);
    cudaError_t attr_error = cudaSuccess;
    std::call_once(once[device & 63], [&] { attr_error = cudaFuncSetAttribute(packed_product_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPackedSmem); });
    GF_CUDA(attr_error);
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(grid);
    config.blockDim = dim3(kPackedThreads);
    config.dynamicSmemBytes = kPackedSmem;
    config.stream = stream;
    cudaLaunchAttribute attribute;
    attribute.id = cudaLaunchAttributeCooperative;
    attribute.val.cooperative = 1;
    config.attrs = &attribute;
    config.numAttrs = 1;
    GF_CUDA(cudaLaunchKernelEx(&config, packed_product_kernel, p));
    return GF_OK;
}

}  // namespace gf
