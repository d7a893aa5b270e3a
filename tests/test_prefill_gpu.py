"""Prompt ingestion on the tensor cores: the 256-row bf16 GEMM (two 128-row products per dequantised weight tile) with in-kernel dequantisation
(tcgen05 / TMEM) against the CPU oracle, and chunked prefill against token-at-a-time decoding."""
import numpy as np
import pytest

from guffin_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


def bf16_round(a):
    """Round-to-nearest-even to bfloat16, returned as float32."""
    bits = np.ascontiguousarray(a, np.float32).view(np.uint32).astype(np.uint64)
    bits = (bits + 0x7fff + ((bits >> 16) & 1)) & 0xffff0000
    return bits.astype(np.uint32).view(np.float32)


def rel_l2(got, want):
    return float(np.linalg.norm(got.astype(np.float64) - want) / max(np.linalg.norm(want), 1e-30))


@pytest.mark.parametrize("dtype,k,n,rows", [(syn.Q4_K, 512, 128, 128), (syn.Q4_K, 3840, 256, 37), (syn.Q6_K, 1024, 384, 128),
                                             (syn.Q6_K, 256, 128, 1), (syn.Q8_0, 640, 256, 100), (syn.Q8_0, 128, 128, 128),
                                             (syn.Q4_K, 15360, 128, 128), (syn.Q4_K, 3840, 256, 200), (syn.Q6_K, 1024, 384, 256),
                                             (syn.Q8_0, 640, 128, 129)])
def test_prefill_matmul_matches_bf16_reference_and_oracle(gf, oracle, dtype, k, n, rows):
    """Against the same product with both operands rounded to bf16 and summed in double precision the
    kernel may differ only by its f32 accumulation (5e-5: a layout or descriptor mistake shows as an
    error of order one); against the f32 oracle by the bf16 rounding of the operands (stated
    tolerance 1e-2 relative L2, measured about 3e-3).  Rows beyond the live ones come back zero."""
    rng = np.random.default_rng(k + n + rows)
    native = syn.make_weight(rng, dtype, k, n)
    weight = gf.PackedWeight(dtype, k, n, native)
    x = rng.standard_normal((rows, k)).astype(np.float32)
    got = gf.prefill_matmul(weight, x)
    assert got.shape == ((rows + 127) // 128 * 128, n)
    w = oracle.dequantize(dtype, native).reshape(n, k)
    exact = bf16_round(x).astype(np.float64) @ bf16_round(w).astype(np.float64).T
    assert rel_l2(got[:rows], exact) < 5e-5                                  # 1.8e-5 at K = 15360: the accumulator does not round to nearest
    assert np.abs(got[:rows] - exact).max() <= 3e-4 * np.abs(exact).max()
    want = oracle.matmul(dtype, x, native, k, n)
    assert rel_l2(got[:rows], want) < 1e-2
    assert not got[rows:].any()
    weight.packed.free()


@pytest.fixture(scope="module")
def gm(gf):
    from guffin_b200 import model
    return model


@pytest.mark.parametrize("geometry,seed", [("tiny-target", 81), ("tiny-draft", 82), ("tiny-gemma2", 83)])
def test_tensor_prefill_matches_exact_row_path(gf, gm, oracle, geometry, seed):
    """A 150-token prompt through the chunked tensor-core path (several chunks, the sliding layers'
    rings wrap) against the exact row path on the same plan geometry: committed K/V rows of every layer
    and the next-token logits agree within the stated bf16 tolerance (operands rounded to 8 bits of
    mantissa in every projection of every layer: 3e-2 relative L2), the positions are equal, and
    decoding continues identically in structure (one more verified pass on both)."""
    from oracle.pyoracle import OracleModel
    config = syn.model_config(geometry)
    weights = syn.make_model_weights(geometry, seed)
    tokens = np.random.default_rng(seed).integers(0, config["vocab"], 160).astype(np.uint32)
    tensor, exact = gm.Model(config, weights, 192, 2), gm.Model(config, weights, 192, 2)
    exact.use_tensor_prefill(False)
    tensor.prefill(tokens[:150])
    exact.prefill(tokens[:150])
    assert tensor.position == exact.position == 150
    assert tensor.prefill_logits_row == 0 and exact.prefill_logits_row == 1          # 150 rows in passes of two
    got, want = tensor.logits(0), exact.logits(1)
    worst_kv = 0.0
    for layer in range(config["layers"]):
        first = 150 - 16                      # rows every layer still holds (the smallest ring keeps 32)
        gk, gv = tensor.read_kv(layer, first, 16)
        wk, wv = exact.read_kv(layer, first, 16)
        worst_kv = max(worst_kv, rel_l2(gk, wk), rel_l2(gv, wv))
    logit_error = rel_l2(got, want)
    print(f"{geometry}: tensor prefill vs exact rows: K/V rel-L2 {worst_kv:.2e}, logits rel-L2 {logit_error:.2e}")
    assert worst_kv < 3e-2 and logit_error < 3e-2
    # The oracle (f32, token at a time) agrees with the tensor path within the same tolerance.
    ref = OracleModel(oracle, config, weights, context=192)
    for token in tokens[:149]:
        ref.append(token, want_logits=False)
    assert rel_l2(got, ref.append(tokens[149])) < 3e-2
    for model in (tensor, exact):
        model.forward(tokens[150:152], logits=True)
        model.publish(2)
        assert model.status() == 0
    assert rel_l2(tensor.logits(1), exact.logits(1)) < 3e-2


@pytest.mark.parametrize("base,rows,window,ring_rows,heads,kv_heads,softcap", [
    (700, 128, 0, 1024, 4, 2, 0.0),         # global layer, a full chunk
    (300, 37, 64, 128, 4, 2, 0.0),          # sliding window inside the ring (wrapped) and into the private rows
    (0, 100, 16, 32, 2, 2, 0.0),            # first chunk of a prompt: private rows only, one head per KV head
    (90, 128, 0, 128, 4, 1, 50.0),          # four heads per KV head, score softcap
    (5, 3, 4, 8, 4, 2, 0.0),                # a few rows
])
def test_prefill_attention_matches_oracle(gf, oracle, base, rows, window, ring_rows, heads, kv_heads, softcap):
    """The chunk attention kernel against the oracle's row attention over each row's logical key
    range (causal, sliding window including the row itself, ring slots overwritten by later
    positions): f16 queries and softmax weights on the tensor cores, tolerance 2e-3."""
    L = gf.load()
    hd, kvw = 256, kv_heads * 256
    rng = np.random.default_rng(base + rows)
    keys = rng.standard_normal((base + rows, kvw)).astype(np.float16)
    values = rng.standard_normal((base + rows, kvw)).astype(np.float16)
    q = rng.standard_normal((rows, heads * hd)).astype(np.float32)
    ring_k, ring_v = np.zeros((ring_rows, kvw), np.float16), np.zeros((ring_rows, kvw), np.float16)
    for p in range(base):
        ring_k[p & (ring_rows - 1)], ring_v[p & (ring_rows - 1)] = keys[p], values[p]
    bufs = [gf.DeviceBuffer.from_numpy(np.ascontiguousarray(a)) for a in (q, ring_k, ring_v, keys[base:], values[base:])]
    out = gf.DeviceBuffer(q.nbytes)
    pos = gf.DeviceBuffer.from_numpy(np.array([base], np.uint32))
    gf.check(L.gf_prefill_attention(bufs[0].ptr, bufs[1].ptr, bufs[2].ptr, bufs[3].ptr, bufs[4].ptr, out.ptr, pos.ptr,
                                    rows, heads, kv_heads, hd, ring_rows, window, 0.0625, softcap, None))
    gf.check(L.gf_stream_synchronize(None))
    got = out.download(np.float32).reshape(rows, -1)
    for r in range(rows):
        p = base + r
        first = max(0, p + 1 - window) if window else 0
        want = oracle.attention_row(q[r], keys[first:p + 1].astype(np.float32), values[first:p + 1].astype(np.float32),
                                    heads, kv_heads, hd, 0.0625, softcap)
        assert np.abs(got[r] - want).max() <= 2e-3 * max(1.0, np.abs(want).max()), (base, r, window)


@pytest.mark.parametrize("base,rows,window,ring_rows,heads,kv_heads,softcap", [
    (0, 1, 0, 8, 2, 1, 0.0),                # one row at the first position: one tile of one key
    (63, 65, 0, 64, 4, 4, 0.0),             # tile and block borders, one head per KV head
    (190, 256, 100, 256, 4, 2, 0.0),        # windows that begin inside tiles
    (30, 129, 64, 64, 4, 1, 30.0),          # four heads per KV head, a window of a whole tile
    (500, 40, 1, 512, 2, 2, 0.0),           # every row sees itself alone
])
def test_prefill_attention_borders(gf, oracle, base, rows, window, ring_rows, heads, kv_heads, softcap):
    """Borders of the 128-query blocks and 64-key tiles, for every way heads share a block."""
    test_prefill_attention_matches_oracle(gf, oracle, base, rows, window, ring_rows, heads, kv_heads, softcap)


@pytest.mark.parametrize("geometry,seed,cuts", [
    ("tiny-target", 84, (300, 257)),        # rings of 32 rows that a chunk overflows; a second chunk behind a filled ring
    ("tiny-target", 85, (65, 2100)),        # a short chunk ahead, then two equal wide ones
    ("tiny-draft", 86, (330, 700)),         # an f32 cache: Q8_0 weights, chunks limited to 1024 rows
    ("tiny-gemma2", 87, (511, 300)),        # capped scores, no norms of the heads
    ("tiny-target", 88, (66, 97, 257)),     # chunks of up to 256 rows, decoded on their way to the tensor core: the shortest,
    ("tiny-draft", 89, (225, 130)),         # products of 96, 128, 160, 224 and 256 rows
    ("tiny-gemma2", 90, (161, 193)),
])
def test_wide_prompt_chunks(gf, gm, geometry, seed, cuts):
    """Chunks of more than 256 rows (weights decoded to HBM, products on pairs of CTAs) and shorter ones against the exact row path: K/V rows
    and logits within the bound the 256-row chunks have (test_tensor_prefill_matches_exact_row_path), and decoding behind them."""
    config = syn.model_config(geometry)
    weights = syn.make_model_weights(geometry, seed)
    total = sum(cuts)
    tokens = np.random.default_rng(seed).integers(0, config["vocab"], total + 2).astype(np.uint32)
    wide, exact = gm.Model(config, weights, total + 64, 8), gm.Model(config, weights, total + 64, 8)
    exact.use_tensor_prefill(False)
    for model in (wide, exact):
        done = 0
        for count in cuts:
            model.prefill(tokens[done:done + count])
            done += count
        assert model.position == total and model.status() == 0
    worst = rel_l2(wide.logits(0), exact.logits(exact.prefill_logits_row))
    for layer in range(config["layers"]):
        for got, want in zip(wide.read_kv(layer, total - 12, 12), exact.read_kv(layer, total - 12, 12)):
            worst = max(worst, rel_l2(got, want))
    print(f"{geometry} {cuts}: wide chunks vs exact rows {worst:.2e}")
    assert worst < 3e-2
    for model in (wide, exact):
        model.forward(tokens[total:], logits=True)
        model.publish(2)
        model.truncate(total)
        assert model.status() == 0
    assert rel_l2(wide.logits(1), exact.logits(1)) < 3e-2


@pytest.mark.parametrize("geometry,ffn,rows", [("tiny-target", 16384, 66), ("tiny-target", 20736, 200), ("tiny-draft", 24576, 131)])
def test_tiles_cut_between_ctas(gf, gm, geometry, ffn, rows):
    """A down projection of few columns and long K, whose tiles are cut along K and added from pieces, and gate and up
    products of more tiles than SMs, some of them cut: K/V rows and logits against the exact row path, twice in a row."""
    config = dict(syn.model_config(geometry), ffn=ffn, layers=2)
    weights = syn.make_model_weights(geometry, 91, config)
    tokens = np.random.default_rng(91).integers(0, config["vocab"], rows + 1).astype(np.uint32)
    tensor, exact = gm.Model(config, weights, rows + 32, 8), gm.Model(config, weights, rows + 32, 8)
    exact.use_tensor_prefill(False)
    exact.prefill(tokens)
    for _ in range(2):
        tensor.reset()
        tensor.prefill(tokens)
        assert tensor.status() == 0
        worst = rel_l2(tensor.logits(0), exact.logits(exact.prefill_logits_row))
        for layer in range(2):
            for got, want in zip(tensor.read_kv(layer, rows - 8, 8), exact.read_kv(layer, rows - 8, 8)):
                worst = max(worst, rel_l2(got, want))
        assert worst < 3e-2


@pytest.mark.parametrize("geometry,row_capacity,count", [("tiny-target", 1, 9), ("tiny-target", 2, 10), ("tiny-target", 3, 47),
                                                         ("tiny-draft", 2, 64), ("tiny-gemma2", 8, 33)])
def test_short_prompts_in_wide_passes(gf, gm, geometry, row_capacity, count):
    """A prompt too short for chunks runs in passes of eight rows whatever the plan's passes hold, the last pass in the
    plan's own: cache rows, logits and the last pass taken back and run again, against tokens given one by one.  Products do not
    depend on the rows of a pass; the attention's partitions do, by f32 roundings that binary16 cache rows (2^-11) amplify."""
    config = syn.model_config(geometry)
    weights = syn.make_model_weights(geometry, 92)
    tokens = np.random.default_rng(92).integers(0, config["vocab"], count).astype(np.uint32)
    plan, single = gm.Model(config, weights, 80, row_capacity), gm.Model(config, weights, 80, 1)
    plan.prefill(tokens)
    for token in tokens:
        single.forward(np.array([token], np.uint32), logits=True)
        single.publish(1)
    assert plan.position == count and plan.status() == 0
    assert plan.prefill_logits_row < row_capacity
    assert rel_l2(plan.logits(plan.prefill_logits_row), single.logits(0)) < 2e-3
    for layer in range(config["layers"]):
        for got, want in zip(plan.read_kv(layer, count - 8, 8), single.read_kv(layer, count - 8, 8)):
            assert rel_l2(got, want) < 2e-3
    plan.truncate(count - row_capacity)
    plan.forward(tokens[count - row_capacity:], logits=True)
    assert rel_l2(plan.logits(row_capacity - 1), single.logits(0)) < 2e-3
