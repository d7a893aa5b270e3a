// Prompt chunks of up to kWideRows rows of a quantised plan: a launch's weights are decoded to bf16 tiles in HBM once and
// multiplied with all rows of the chunk by the product kernel of the layered plans (dense_prefill.cu), norms, rotation and
// gate fused around it (Model::prefill_wide, model.cu).  2048 tokens into the 12B plan: 131.8 ms in chunks of 256 rows of prefill.cu's
// kernel (which decodes in shared memory), 45.2 ms in one of 2048; 777 tokens into the 270M plan 5.1 -> 3.3 ms.
#pragma once

#include "dense.cuh"
#include "ops.cuh"

namespace gf {

constexpr uint32_t kWideRows = 2048;

// One matrix of a launch: its packed weights and where its decoded tiles begin.  Groups of eight columns go to group
// (n / 8) * group_step + group_first (step 2: one half of a gate / up pair).
struct WideMatrix {
    const uint8_t* packed;
    uint8_t* tiles;
    uint32_t dtype, pairs, units, k_blocks, group_step, group_first, first_warp;
};
struct WideDecode {
    WideMatrix m[3];
    uint32_t matrices = 0, warps = 0;
};
// The reference's values exactly, then one rounding to bf16 (as prefill.cu's kernel decodes them).
int launch_wide_decode(const WideDecode& decode, cudaStream_t stream);

// Chunks of up to kPackedRows rows instead decode a launch's weights on their way to the tensor core (packed_product.cu).
constexpr uint32_t kPackedRows = 256;
struct PackedProduct {
    struct Matrix {
        const uint8_t* packed = nullptr;
        float* out = nullptr;                    // [rows][n]; not used by a pair
        uint32_t dtype = 0, n = 0, first_tile = 0;
    } m[3];
    uint32_t matrices = 0, rows = 0, k = 0;
    bool paired = false;                         // two matrices of one shape: result(row, n) = gelu(m[0]) * m[1]
    Operand a, result;
    float* partial = nullptr;                    // packed_partial_bytes()
    uint32_t* counters = nullptr;                // two per 128 columns of the launch, zero between launches
    int* error_flag = nullptr;
    uint32_t tiles = 0, units = 0, unit_elems = 0, n_rows = 0, row_bytes = 0, stages = 0, unit_slots = 0;      // filled by the launcher
};
size_t packed_partial_bytes();
int launch_packed_product(PackedProduct product, cudaStream_t stream);

// Per-head norm (skipped without weights), rotation from the table, and the cache rows: q [rows][heads * 256] f16
// multiplied by `scale` (or f32 as it is, with q32), keys and values [rows][kv_heads * 256] f16 or f32.
struct WideRope {
    const float *raw_q, *raw_k, *raw_v;          // raw_q may be null: keys and values only
    const float *q_norm, *k_norm;
    __half* q;
    float* q32;
    void *keys, *values;
    const uint32_t* position;                    // of row 0
    const float2* rotation;                      // [table_rows][128]
    uint32_t* status;
    uint32_t rows, heads, kv_heads, table_rows;
    float eps, scale;
    int kv_f16;
};
int launch_wide_rope(const WideRope& rope, cudaStream_t stream);

// Rows [first, rows) of a chunk's own cache rows into their ring slots.
int launch_wide_publish(const void* own_k, const void* own_v, void* ring_k, void* ring_v, const uint32_t* position, uint32_t first, uint32_t rows,
                        uint32_t ring_mask, uint32_t row_bytes, cudaStream_t stream);
int launch_advance_position(uint32_t* position, uint32_t rows, cudaStream_t stream);

}  // namespace gf
