// Kernels of wide prompt chunks (see prompt.cuh).
#include "prompt.cuh"
#include "dequant_bf16.cuh"

namespace gf {

namespace {

// A warp decodes one pair row (16 columns x one K unit): 2.3-3.4 KB in, 8 KB (Q8_0: 4 KB) out, 256 contiguous bytes per
// store.  Bound by HBM (what it reads and writes).
__global__ void __launch_bounds__(256) wide_decode_kernel(const __grid_constant__ WideDecode p) {
    const uint32_t lane = threadIdx.x & 31u, item = blockIdx.x * 8u + (threadIdx.x >> 5);
    if (item >= p.warps) return;
    uint32_t which = 0;
    while (which + 1u < p.matrices && item >= p.m[which + 1u].first_warp) ++which;
    const WideMatrix& m = p.m[which];
    const uint32_t at = item - m.first_warp, pair = at / m.units, unit = at % m.units;
    const uint8_t* row = m.packed + (size_t)at * pair_row_bytes((int)m.dtype);      // pair rows of a pair lie behind one another
    const uint32_t subs = m.dtype == GF_Q8_0 ? 2u : 4u;
#pragma unroll
    for (uint32_t half = 0; half < 2u; ++half) {
        const uint32_t group = (2u * pair + half) * m.group_step + m.group_first, column = (group % 16u) * 8u + (lane >> 2);
        uint8_t* tile = m.tiles + ((size_t)(group / 16u) * m.k_blocks + unit * subs) * kDenseTileBytes;
        if (m.dtype == GF_Q4_K) {
#pragma unroll
            for (uint32_t sub = 0; sub < 4u; ++sub) dequant_q4k(row, sub, lane, half, column, tile + sub * kDenseTileBytes);
        } else if (m.dtype == GF_Q6_K) {
#pragma unroll
            for (uint32_t sub = 0; sub < 4u; ++sub) dequant_q6k(row, sub, lane, half, column, tile + sub * kDenseTileBytes);
        } else {
#pragma unroll
            for (uint32_t sub = 0; sub < 2u; ++sub) dequant_q80(row, sub, lane, half, column, tile + sub * kDenseTileBytes);
        }
    }
}

// A warp per (row, head): lane l holds dimensions 4l .. 4l + 3 and 128 + 4l .. of it, the two halves the rotation pairs.
__global__ void __launch_bounds__(256) wide_rope_kernel(const __grid_constant__ WideRope p) {
    const uint32_t lane = threadIdx.x & 31u, heads = (p.raw_q ? p.heads : 0u) + p.kv_heads;
    const uint32_t item = blockIdx.x * 8u + (threadIdx.x >> 5);
    if (item >= p.rows * heads) return;
    const uint32_t row = item / heads, at = item % heads, queries = heads - p.kv_heads;
    const bool query = at < queries;
    const uint32_t head = query ? at : at - queries;
    const size_t from = query ? ((size_t)row * p.heads + head) * 256u : ((size_t)row * p.kv_heads + head) * 256u;
    const float* src = (query ? p.raw_q : p.raw_k) + from;
    const float* gain = query ? p.q_norm : p.k_norm;
    auto load = [&](const float* x, float (&v)[8]) {
        const float4 a = *reinterpret_cast<const float4*>(x + 4u * lane), b = *reinterpret_cast<const float4*>(x + 128u + 4u * lane);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    };
    float v[8];
    load(src, v);
    if (gain) {
        float total = 0.0f, g[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) total = fmaf(v[i], v[i], total);
        total = warp_sum(total);
        load(gain, g);
        const float inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(total, 256.0f), p.eps)));
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = __fmul_rn(__fmul_rn(v[i], inv), g[i]);
    }
    const uint32_t position = min(*p.position + row, p.table_rows - 1u);
    const float4* turn = reinterpret_cast<const float4*>(p.rotation + (size_t)position * 128u + 4u * lane);      // two (cos, sin) pairs each
    const float4 t0 = turn[0], t1 = turn[1];
    const float c[4] = {t0.x, t0.z, t1.x, t1.z}, s[4] = {t0.y, t0.w, t1.y, t1.w};
    float r[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        r[i] = __fsub_rn(__fmul_rn(v[i], c[i]), __fmul_rn(v[i + 4], s[i]));
        r[i + 4] = __fadd_rn(__fmul_rn(v[i], s[i]), __fmul_rn(v[i + 4], c[i]));
    }
    bool finite = true;
    auto store_half = [&](__half* to, const float (&x)[8], float scale) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            __half2 w[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                w[i] = __floats2half2_rn(x[4 * h + 2 * i] * scale, x[4 * h + 2 * i + 1] * scale);
                finite = finite && isfinite(__low2float(w[i])) && isfinite(__high2float(w[i]));
            }
            *reinterpret_cast<uint2*>(to + 128 * h + 4u * lane) = *reinterpret_cast<const uint2*>(w);
        }
    };
    auto store = [&](float* to, const float (&x)[8]) {
        *reinterpret_cast<float4*>(to + 4u * lane) = make_float4(x[0], x[1], x[2], x[3]);
        *reinterpret_cast<float4*>(to + 128u + 4u * lane) = make_float4(x[4], x[5], x[6], x[7]);
    };
    if (query) {
        if (p.q) store_half(p.q + from, r, p.scale);
        else store(p.q32 + from, r);
        return;
    }
    float value[8];
    load(p.raw_v + from, value);
    if (p.kv_f16) {
        store_half(static_cast<__half*>(p.keys) + from, r, 1.0f);
        store_half(static_cast<__half*>(p.values) + from, value, 1.0f);
        if (!finite) atomicOr(p.status, kStatusKvNonFinite);
    } else {
        store(static_cast<float*>(p.keys) + from, r);
        store(static_cast<float*>(p.values) + from, value);
    }
}

__global__ void __launch_bounds__(128) wide_publish_kernel(const uint8_t* own_k, const uint8_t* own_v, uint8_t* ring_k, uint8_t* ring_v, const uint32_t* position,
                                                           uint32_t first, uint32_t ring_mask, uint32_t row_bytes) {
    const uint32_t row = first + blockIdx.x;
    const size_t dst = (size_t)((*position + row) & ring_mask) * row_bytes, src = (size_t)row * row_bytes;
    for (uint32_t b = threadIdx.x * 16u; b < row_bytes; b += blockDim.x * 16u) {
        *reinterpret_cast<uint4*>(ring_k + dst + b) = *reinterpret_cast<const uint4*>(own_k + src + b);
        *reinterpret_cast<uint4*>(ring_v + dst + b) = *reinterpret_cast<const uint4*>(own_v + src + b);
    }
}

__global__ void advance_kernel(uint32_t* position, uint32_t rows) {
    if (threadIdx.x == 0) position[0] += rows;
}

}  // namespace

int launch_wide_decode(const WideDecode& decode, cudaStream_t stream) {
    if (decode.matrices == 0 || decode.warps == 0) return fail(GF_ERR_INVALID, "wide decode: nothing to decode");
    wide_decode_kernel<<<(decode.warps + 7u) / 8u, 256, 0, stream>>>(decode);
    GF_CUDA(cudaGetLastError());
    return GF_OK;
}

int launch_wide_rope(const WideRope& p, cudaStream_t stream) {
    if (!p.raw_k || !p.raw_v || !p.keys || !p.values || !p.rotation || (p.raw_q && !p.q && !p.q32)) return fail(GF_ERR_INVALID, "wide rope: bad arguments");
    const uint32_t items = p.rows * ((p.raw_q ? p.heads : 0u) + p.kv_heads);
    wide_rope_kernel<<<(items + 7u) / 8u, 256, 0, stream>>>(p);
    GF_CUDA(cudaGetLastError());
    return GF_OK;
}

int launch_wide_publish(const void* own_k, const void* own_v, void* ring_k, void* ring_v, const uint32_t* position, uint32_t first, uint32_t rows,
                        uint32_t ring_mask, uint32_t row_bytes, cudaStream_t stream) {
    wide_publish_kernel<<<rows - first, 128, 0, stream>>>(static_cast<const uint8_t*>(own_k), static_cast<const uint8_t*>(own_v), static_cast<uint8_t*>(ring_k),
                                                          static_cast<uint8_t*>(ring_v), position, first, ring_mask, row_bytes);
    GF_CUDA(cudaGetLastError());
    return GF_OK;
}

int launch_advance_position(uint32_t* position, uint32_t rows, cudaStream_t stream) {
    advance_kernel<<<1, 32, 0, stream>>>(position, rows);
    GF_CUDA(cudaGetLastError());
    return GF_OK;
}

}  // namespace gf
