// Causal attention of a prompt chunk over keys and values per head or per group of heads, binary16 (see latent.cuh).
#include "grouped.cuh"
#include "latent.cuh"
#include "tcgen05.cuh"

#include <mutex>

namespace gf {

namespace {

constexpr uint32_t kRows = 128, kKeys = 64;                            // queries of a block, keys of a tile
constexpr uint32_t kSoftmaxWarps = 4, kIssuingWarp = 4, kCopyWarps = 3, kThreads = (kSoftmaxWarps + 1u + kCopyWarps) * 32u;
constexpr uint32_t kWeightBytes = kRows * kKeys * 2u;                  // softmax weights of a tile, f16
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kSlack = 8.0f;                                         // factors of two by which a row's maximum may lag

__device__ __forceinline__ void copy16(void* dst_smem, const void* src, bool valid) {      // zero-fills when not valid
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst_smem)), "l"(src), "r"(valid ? 16u : 0u) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void arrive(uint64_t* bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory"); }
__device__ __forceinline__ uint32_t half_pair(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float power_of_two(float x) {              // 2 ulp; results below 2^-126 are zero
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Block = 128 queries (128 / pack chunk rows x `pack` heads of one key/value head) on the tensor core: scores of a tile
// of 64 keys (M = 128, N = 64), softmax in registers, outputs (M = 128, N = vdim_pad, K = 64) accumulated in tensor memory.
// Every operand lies in shared memory as core matrices of eight rows x 16 bytes; a tile of values, stored like one of
// keys, is the product's B operand with its rows contiguous.
//
// Warps 0-3: a thread has a query.  It keeps the scores' running maximum and sum, writes the weights as the next product's
// A operand, and rescales the outputs only when its maximum has grown by more than 2^kSlack since it last did (weights are
// then up to 2^8; sums and outputs share the factor).  Warp 4 issues: the scores of tile i + 1 before the outputs of tile
// i, so that the tensor core works under the softmax.  Warps 5-7 copy keys and values, two tiles of either in flight.
//
// Bound by the softmax for heads up to 128 (about 1000 cycles a tile against 512 of the tensor core; two blocks share an
// SM), by the tensor core above (1024 cycles).  It replaced a mma.sync kernel of 64 x 64 tiles that ran at 97 TFLOP/s for
// 128-wide heads: prompts of eight layers 4.24 -> 3.81 ms (2048 tokens, 16 heads) and 2.47 -> 2.33 ms (1500 tokens, four
// of the layers attend).  kCap: capped scores.  kBlocks: blocks of an SM.
template <bool kCap, int kBlocks>
__global__ void __launch_bounds__(kThreads, kBlocks) head_attention_kernel(const __grid_constant__ HeadAttention p, const uint32_t pack) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint32_t tmem_slot, abort_flag;
    __shared__ __align__(8) uint64_t keys_full[2], keys_free[2], values_full[2], outputs_done[2], scores_full[2], scores_free[2], weights_full;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t dim = p.dim_pad, vdim = p.vdim_pad, key_bytes = kKeys * dim * 2u, value_bytes = kKeys * vdim * 2u;
    uint8_t* q_tile = smem;                                            // [128] x dim
    uint8_t* weights = q_tile + kRows * dim * 2u;                      // [128] x 64
    uint8_t* k_tiles = weights + kWeightBytes;                         // two of [64] x dim
    uint8_t* v_tiles = k_tiles + 2u * key_bytes;                       // two of [64] x vdim
    const volatile uint32_t* abort = &abort_flag;

    // Queries of this block: rows first_row .. of heads first_head .. + pack.
    const uint32_t block_rows = kRows / pack, share = p.heads / p.kv_heads;
    const uint32_t first_row = (gridDim.x - 1u - blockIdx.x) * block_rows, first_head = blockIdx.y * pack, kv = first_head / share;      // the longest blocks first
    const uint32_t base = *p.position, end = base + min(first_row + block_rows, p.rows);
    const uint32_t from = p.window != 0u && base + first_row + 1u > p.window ? base + first_row + 1u - p.window : 0u;
    const uint32_t tiles = (end - from + kKeys - 1u) / kKeys;

    if (tid == 0) {
        abort_flag = 0u;
        for (uint32_t i = 0; i < 2u; ++i) {
            mbar_init(&keys_full[i], kCopyWarps); mbar_init(&values_full[i], kCopyWarps); mbar_init(&keys_free[i], 1);
            mbar_init(&outputs_done[i], 1); mbar_init(&scores_full[i], 1); mbar_init(&scores_free[i], kSoftmaxWarps);
        }
        mbar_init(&weights_full, kSoftmaxWarps);
        fence_barrier_init();
    }
    const uint32_t columns = kBlocks == 1 ? 512u : 256u;               // two sets of 64 score columns, then the outputs
    __syncwarp();
    if (warp == 0) tmem_alloc(&tmem_slot, columns);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = tmem_slot, outputs = tmem + 2u * kKeys;
    bool ok = true;

    if (warp > kIssuingWarp) {
        // ---- copies.  A lane has key lane % 8 of a group of eight, and every fourth of its 16-byte pieces.
        const uint32_t w = warp - kIssuingWarp - 1u, eighth = lane & 7u, piece0 = lane >> 3;
        const uint32_t own_from = p.rings || p.ring_k ? base : 0u;     // keys before the chunk lie in the rings, or ahead of the chunk's own where there are none
        const __half *ring_k = p.ring_k, *ring_v = p.ring_v;
        if (p.rings) { ring_k = static_cast<const __half*>(p.rings->ring_k); ring_v = static_cast<const __half*>(p.rings->ring_v); }
        if (ring_k) { ring_k += (size_t)kv * dim; ring_v += (size_t)kv * vdim; }
        const __half *own_k = p.k + (size_t)kv * dim, *own_v = p.v + (size_t)kv * vdim;
        auto copy_rows = [&](uint8_t* to, uint32_t tile, const __half* ring, const __half* own, uint32_t width) {
            const size_t ld = (size_t)p.kv_heads * width;
            for (uint32_t group = w; group < kKeys / 8u; group += kCopyWarps) {
                const uint32_t position = from + tile * kKeys + group * 8u + eighth;
                const bool valid = position < end, cached = position < own_from;
                const __half* src = !valid ? own : cached ? ring + (size_t)(position & p.ring_mask) * ld : own + (size_t)(position - own_from) * ld;
                uint8_t* dst = to + group * width * 16u + eighth * 16u;
                for (uint32_t piece = piece0; piece < width / 8u; piece += 4u) copy16(dst + piece * 128u, src + piece * 8u, valid);
            }
        };
        for (uint32_t group = w; group < kRows / 8u; group += kCopyWarps) {
            const uint32_t m = group * 8u + eighth, row = first_row + m / pack, head = first_head + m % pack;
            const bool valid = row < p.rows;
            const size_t from_q = ((size_t)(valid ? row : 0u) * p.heads + head) * dim;
            uint8_t* dst = q_tile + group * dim * 16u + eighth * 16u;
            if (!p.q32) {
                for (uint32_t piece = piece0; piece < dim / 8u; piece += 4u) copy16(dst + piece * 128u, p.q + from_q + piece * 8u, valid);
                continue;
            }
            for (uint32_t piece = piece0; piece < dim / 8u; piece += 4u) {
                const float4 x = *reinterpret_cast<const float4*>(p.q32 + from_q + piece * 8u), y = *reinterpret_cast<const float4*>(p.q32 + from_q + piece * 8u + 4u);
                const float scale = p.q_scale;
                *reinterpret_cast<uint4*>(dst + piece * 128u) = valid ? make_uint4(half_pair(x.x * scale, x.y * scale), half_pair(x.z * scale, x.w * scale),
                                                                                   half_pair(y.x * scale, y.y * scale), half_pair(y.z * scale, y.w * scale))
                                                                      : make_uint4(0u, 0u, 0u, 0u);
            }
        }
        uint64_t* due = nullptr;                                       // barrier of the copies requested last but not told of yet
        auto tell = [&]() {
            fence_async_smem();
            __syncwarp();
            if (lane == 0) arrive(due);
        };
        auto request = [&](uint64_t* free, uint32_t parity, uint64_t* full, auto copy) {
            if (!__all_sync(0xffffffffu, mbar_try_wait(free, parity))) {
                if (due) { copies_wait<0>(); tell(); due = nullptr; }
                if (__any_sync(0xffffffffu, !wait_or_abort(free, parity, abort))) return false;
            }
            copy();
            copies_commit();
            if (due) { copies_wait<1>(); tell(); }
            due = full;
            return true;
        };
        for (uint32_t i = 0; i < tiles && ok; ++i) {
            const uint32_t slot = i & 1u, parity = ((i >> 1) & 1u) ^ 1u;      // of the use before; the first use of a barrier passes
            ok = request(&keys_free[slot], parity, &keys_full[slot], [&] { copy_rows(k_tiles + slot * key_bytes, i, ring_k, own_k, dim); })
                 && request(&outputs_done[slot], parity, &values_full[slot], [&] { copy_rows(v_tiles + slot * value_bytes, i, ring_v, own_v, vdim); });
        }
        copies_wait<0>();
        if (due) tell();
        if (!ok && lane == 0) abort_flag = 1u;
    } else if (warp == kIssuingWarp) {
        // ---- products
        const uint64_t q_first = operand_descriptor(smem_u32(q_tile), 128u, dim * 16u), k_first = operand_descriptor(smem_u32(k_tiles), 128u, dim * 16u);
        const uint64_t w_first = operand_descriptor(smem_u32(weights), 128u, kKeys * 16u), v_first = operand_descriptor(smem_u32(v_tiles), vdim * 16u, 128u);
        const uint32_t score_instruction = mma_instruction_f16(kRows, kKeys), output_instruction = mma_instruction_f16(kRows, vdim, kMmaRowsOfB);
        auto scores = [&](uint32_t i) {
            const uint32_t slot = i & 1u, parity = (i >> 1) & 1u;
            if (!wait_or_abort(&keys_full[slot], parity, abort) || !wait_or_abort(&scores_free[slot], parity ^ 1u, abort)) return false;
            tc_fence_after_sync();
            if (elect_one()) {
                for (uint32_t kk = 0; kk < dim / 16u; ++kk)
                    mma_bf16(tmem + slot * kKeys, q_first + kk * 16u, k_first + slot * (key_bytes / 16u) + kk * 16u, score_instruction, kk != 0u ? 1u : 0u);
                mma_commit(&scores_full[slot]);
                mma_commit(&keys_free[slot]);
            }
            __syncwarp();
            return true;
        };
        ok = scores(0);
        for (uint32_t i = 0; i < tiles && ok; ++i) {
            const uint32_t slot = i & 1u;
            if (i + 1u < tiles && !scores(i + 1u)) { ok = false; break; }
            if (!wait_or_abort(&values_full[slot], (i >> 1) & 1u, abort) || !wait_or_abort(&weights_full, i & 1u, abort)) { ok = false; break; }
            tc_fence_after_sync();
            if (elect_one()) {
#pragma unroll
                for (uint32_t kk = 0; kk < kKeys / 16u; ++kk)
                    mma_bf16(outputs, w_first + kk * 16u, v_first + slot * (value_bytes / 16u) + kk * 2u * vdim, output_instruction, (i | kk) != 0u ? 1u : 0u);
                mma_commit(&outputs_done[slot]);
            }
            __syncwarp();
        }
        if (!ok && lane == 0) abort_flag = 1u;
    } else {
        // ---- softmax: this thread's query
        const uint32_t row = first_row + tid / pack, head = first_head + tid % pack, lanes = (warp * 32u) << 16;
        const bool live = row < p.rows;
        const uint32_t last = live ? base + row : 0u;                  // positions it sees; a query that does not exist sees none
        const uint32_t first = !live ? 1u : p.window != 0u && last + 1u > p.window ? last + 1u - p.window : 0u;
        float top = -INFINITY, sum = 0.0f;                             // top: in factors of two
        const float inverse_cap = kCap ? 1.0f / p.softcap : 0.0f;
        uint8_t* mine = weights + (tid >> 3) * (kKeys * 16u) + (tid & 7u) * 16u;
        for (uint32_t i = 0; i < tiles; ++i) {
            const uint32_t slot = i & 1u, at = from + i * kKeys;
            if (__any_sync(0xffffffffu, !wait_or_abort(&scores_full[slot], (i >> 1) & 1u, abort))) { ok = false; break; }
            tc_fence_after_sync();
            float s[2][32];
            tmem_load_32(tmem + lanes + slot * kKeys, s[0]);
            tmem_load_32(tmem + lanes + slot * kKeys + 32u, s[1]);
            tc_fence_before_sync();
            if (lane == 0) arrive(&scores_free[slot]);
            if (kCap)
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int j = 0; j < 32; ++j) s[h][j] = soft_cap(s[h][j], p.softcap, inverse_cap);
            if (__any_sync(0xffffffffu, at < first || at + kKeys > last + 1u))      // some query does not see some key of the tile
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        if (at + h * 32 + j < first || at + h * 32 + j > last) s[h][j] = -INFINITY;
            float most[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int j = 0; j < 32; ++j) most[j & 3] = fmaxf(most[j & 3], s[h][j]);
            float now = fmaxf(fmaxf(most[0], most[1]), fmaxf(most[2], most[3]));
            now *= kLog2e;
            // The outputs so far, and with them the weights' buffer, are not touched by a product any more.
            if (i > 0u) {
                const uint32_t before = i - 1u;
                if (__any_sync(0xffffffffu, !wait_or_abort(&outputs_done[before & 1u], (before >> 1) & 1u, abort))) { ok = false; break; }
                tc_fence_after_sync();
            }
            const bool grown = now > top + kSlack || (top == -INFINITY && now > top);
            const float factor = grown ? power_of_two(top - now) : 1.0f;
            if (grown) { top = now; sum *= factor; }
            if (i > 0u && __any_sync(0xffffffffu, grown)) {
                for (uint32_t c = 0; c < vdim; c += 16u) {
                    float o[16];
                    tmem_load_16(outputs + lanes + c, o);
#pragma unroll
                    for (int j = 0; j < 16; ++j) o[j] *= factor;
                    tmem_store_16(outputs + lanes + c, o);
                }
            }
            const float shift = top == -INFINITY ? 0.0f : top;
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    float w[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) w[j] = power_of_two(fmaf(s[h][c * 8 + j], kLog2e, -shift));
                    sum += ((w[0] + w[1]) + (w[2] + w[3])) + ((w[4] + w[5]) + (w[6] + w[7]));
                    *reinterpret_cast<uint4*>(mine + (h * 4 + c) * 128) = make_uint4(half_pair(w[0], w[1]), half_pair(w[2], w[3]), half_pair(w[4], w[5]), half_pair(w[6], w[7]));
                }
            fence_async_smem();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) arrive(&weights_full);
        }
        const uint32_t before = tiles - 1u;
        if (ok && __any_sync(0xffffffffu, !wait_or_abort(&outputs_done[before & 1u], (before >> 1) & 1u, abort))) ok = false;
        if (!ok && lane == 0) abort_flag = 1u;
        if (ok) {
            tc_fence_after_sync();
            float factor = 1.0f / sum;
            if (p.sink && live) {
                const float sink = p.sink[head] * kLog2e, most = fmaxf(top, sink);
                factor = exp2f(top - most) / (sum * exp2f(top - most) + exp2f(sink - most));
            }
            if (p.gate && live) factor *= sigmoid(p.gate[(size_t)row * p.heads + head]);
            for (uint32_t c = 0; c < vdim; c += 16u) {
                float o[16];
                tmem_load_16(outputs + lanes + c, o);
                if (!live) continue;
                const uint32_t column = head * p.vdim + c;
                if (c + 16u <= p.vdim && column % 8u == 0u && !p.result.f32) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        uint4 r;
                        uint32_t* word = &r.x;
#pragma unroll
                        for (int j = 0; j < 4; ++j) asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(word[j]) : "f"(o[h * 8 + 2 * j + 1] * factor), "f"(o[h * 8 + 2 * j] * factor));
                        *reinterpret_cast<uint4*>(static_cast<uint8_t*>(p.result.data) + operand_offset(p.result, row, column + h * 8u)) = r;
                    }
                } else if (c + 16u <= p.vdim && column % 4u == 0u && p.result.f32) {
                    float* out = static_cast<float*>(p.result.data) + (size_t)row * p.result.k_pad + column;
#pragma unroll
                    for (int j = 0; j < 16; j += 4) *reinterpret_cast<float4*>(out + j) = make_float4(o[j] * factor, o[j + 1] * factor, o[j + 2] * factor, o[j + 3] * factor);
                } else {
#pragma unroll
                    for (uint32_t j = 0; j < 16u; ++j)
                        if (c + j < p.vdim) store_operand(p.result, row, column + j, o[j] * factor);
                }
            }
            tc_fence_before_sync();
        }
    }
    const bool failed = __syncthreads_or(ok ? 0 : 1) != 0;
    if (failed && tid == 0 && p.error_flag) atomicExch(p.error_flag, 1);
    tc_fence_after_sync();
    if (warp == 0) tmem_dealloc(tmem, columns);
}

// Cache rows [0, positions) -- the ring's, then the chunk's own -- as a bf16 operand.
__global__ void __launch_bounds__(64) latent_operand_kernel(const StreamRings* rings, const __half* __restrict__ own, const uint32_t* __restrict__ base_position,
                                                            uint32_t row_elements, uint32_t ring_mask, const Operand result) {
    const uint32_t position = blockIdx.x, base = *base_position;
    const __half* ring = static_cast<const __half*>(rings->ring_k);
    const __half* src = position < base ? ring + (size_t)(position & ring_mask) * row_elements : own + (size_t)(position - base) * row_elements;
    for (uint32_t piece = threadIdx.x; piece < result.k_pad / 8u; piece += blockDim.x) {
        uint4 out = make_uint4(0u, 0u, 0u, 0u);
        if (piece * 8u < row_elements) {
            const uint4 in = *reinterpret_cast<const uint4*>(src + piece * 8u);
            const __half2* h = reinterpret_cast<const __half2*>(&in);
            uint32_t* o = reinterpret_cast<uint32_t*>(&out);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 f = __half22float2(h[i]);
                asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(o[i]) : "f"(f.y), "f"(f.x));
            }
        }
        *reinterpret_cast<uint4*>(static_cast<uint8_t*>(result.data) + operand_offset(result, position, piece * 8u)) = out;
    }
}

template <bool kCap, int kBlocks>
int launch_instance(const HeadAttention& p, cudaStream_t stream) {
    const uint32_t smem = (kRows + 2u * kKeys) * p.dim_pad * 2u + 2u * kKeys * p.vdim_pad * 2u + kWeightBytes;
    static std::once_flag once[64];
    int device = 0;
    cudaGetDevice(&device);
    cudaError_t error = cudaSuccess;
    std::call_once(once[device & 63], [&] { error = cudaFuncSetAttribute(head_attention_kernel<kCap, kBlocks>, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024 - 1024); });
    GF_CUDA(error);
    // Heads that share keys and values share a block where their number divides its queries.
    const uint32_t share = p.heads / p.kv_heads, pack = kRows % share == 0u ? share : 1u, block_rows = kRows / pack;
    head_attention_kernel<kCap, kBlocks><<<dim3((p.rows + block_rows - 1u) / block_rows, p.heads / pack), kThreads, smem, stream>>>(p, pack);
    GF_CUDA(cudaGetLastError());
    return GF_OK;
}

}  // namespace

int launch_head_attention(const HeadAttention& p, cudaStream_t stream) {
    if ((!p.q && !p.q32) || !p.k || !p.v || (p.result.f32 && p.result.k_pad % 4u) || !p.position || !p.result.data || p.rows == 0 || p.heads == 0 || p.kv_heads == 0 || p.heads % p.kv_heads || p.dim_pad % 16u || p.vdim_pad % 16u || p.dim_pad == 0
        || p.vdim_pad == 0 || p.dim_pad > kHeadAttentionMaxDim || p.vdim_pad > kHeadAttentionMaxDim || p.vdim > p.vdim_pad)
        return fail(GF_ERR_INVALID, "head attention: bad arguments");
    // Two blocks' operands and accumulators fit an SM for heads of up to 128.
    if (p.dim_pad <= 128u && p.vdim_pad <= 128u) return p.softcap > 0.0f ? launch_instance<true, 2>(p, stream) : launch_instance<false, 2>(p, stream);
    return p.softcap > 0.0f ? launch_instance<true, 1>(p, stream) : launch_instance<false, 1>(p, stream);
}

int launch_latent_operand(const StreamRings* rings, const void* own, const uint32_t* position, uint32_t positions, uint32_t row_elements, uint32_t ring_mask,
                          const Operand& result, cudaStream_t stream) {
    if (!rings || !own || !position || positions == 0 || positions > result.capacity || row_elements > result.k_pad || result.f32)
        return fail(GF_ERR_INVALID, "latent operand: bad arguments");
    latent_operand_kernel<<<positions, 64, 0, stream>>>(rings, static_cast<const __half*>(own), position, row_elements, ring_mask, result);
    GF_CUDA(cudaGetLastError());
    return GF_OK;
}

}  // namespace gf
