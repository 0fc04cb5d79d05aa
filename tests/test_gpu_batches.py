"""Products of several activation rows at the sizes where their kernels change path: edges of row
tiles and token groups, super-block counts around the number a CTA splits, and integers at the
ends of their range. Bit-exact against the CPU oracle (batched == per-token,
crates/aot-kernels/tests/dots.rs:205-266)."""
import numpy as np
import pytest

from conftest import assert_bits_equal, make_weights

pytestmark = pytest.mark.gpu

Q4_K, Q5_K, Q6_K = 6, 7, 8


def _run(pkg, ob, ctx, kind, w, xs, m, rows, cols, what):
    q = ob.quantize_act(kind, xs)
    want = ob.matmul(ob.Pool(4), ob.detect_table(), kind, w, q, m, rows, cols)
    dout = ctx.alloc(m * rows * 4)
    ctx.matmul(kind, dout, ctx.to_device(w), ctx.to_device(q.view(np.uint8)), m, rows, cols)
    assert_bits_equal(dout.download(np.float32, m * rows).reshape(m, rows), want, what)
    ctx.device_status()


# All kernels give the same bits, so what ran is asked of the context: launches of the tcgen05 batch kernels.
def _launches(g):
    return g.set_option("kt_launches", 0), g.set_option("qt_launches", 0)


@pytest.fixture(params=["by estimates", "warp level"])
def batch_kernels(pkg, ctx, request):
    """The kernels that a batch gets, and those of mma.sync and of streaming alone."""
    spec = pkg.model.tiny("llama", n_layer=1)
    g = pkg.Gpu(ctx, spec.head, spec.layers, spec.weights, 16, 2)
    alone = request.param == "warp level"
    for name in ("k_tensor", "q80_tensor"):
        g.set_option(name, int(alone))
    before = _launches(g)
    yield g
    if alone:
        assert _launches(g) == before
    for name in ("k_tensor", "q80_tensor"):
        g.set_option(name, 0)
    g.close()


@pytest.mark.parametrize("kind", [Q4_K, Q5_K, Q6_K])
@pytest.mark.parametrize("rows,cols", [(1, 256), (17, 768), (2400, 2304), (4735, 1280)])
def test_k_quant_tile_edges(pkg, ob, ctx, batch_kernels, kind, rows, cols):
    w = make_weights(pkg, kind, rows, cols, 21 + kind + rows, "uniform")
    for m in (3, 8, 9, 17, 64, 65):
        xs = np.random.default_rng(m).standard_normal(m * cols).astype(np.float32)
        _run(pkg, ob, ctx, kind, w, xs, m, rows, cols, f"kind {kind} {rows}x{cols} m {m}")


# Which kernel a small batch takes, by launches: the one-lane kernel is one, kmma_kernel has its
# activations converted first. The two tests around this one rely on kmma_kernel from four rows on.
@pytest.mark.parametrize("kind,rows,cols,m,one_lane", [(Q4_K, 300, 512, 2, True), (Q5_K, 2048, 5376, 2, False), (Q6_K, 2048, 5376, 2, True), (Q4_K, 40, 5376, 2, True),
                                                       (Q6_K, 8200, 256, 3, True), (Q5_K, 8200, 256, 3, False), (Q4_K, 2730, 256, 3, True), (Q6_K, 2731, 256, 3, False), (Q6_K, 1, 256, 4, False),
                                                       (Q4_K, 17, 768, 4, False), (Q6_K, 48, 1024, 12, False)])
def test_k_quant_small_batches(pkg, ob, ctx, kind, rows, cols, m, one_lane):
    spec = pkg.model.tiny("llama", n_layer=1)
    g = pkg.Gpu(ctx, spec.head, spec.layers, spec.weights, 16, 2)  # for the count of launches
    w = make_weights(pkg, kind, rows, cols, 23 + kind, "uniform")
    before = g.dispatches()
    _run(pkg, ob, ctx, kind, w, np.random.default_rng(m).standard_normal(m * cols).astype(np.float32), m, rows, cols, f"kind {kind} {rows}x{cols} m {m}")
    assert g.dispatches() - before == (1 if one_lane else 2)
    g.close()


@pytest.mark.parametrize("kind", [Q4_K, Q5_K, Q6_K])
def test_k_quant_integers_at_their_bounds(pkg, ob, ctx, batch_kernels, kind):
    rows, cols, m = 48, 1024, 12
    w = make_weights(pkg, kind, rows, cols, 5, "uniform").reshape(rows * cols // 256, -1)
    w[:, 4:] = 0xFF                                   # largest quants, scales and mins (Q4_K, Q5_K)
    if kind == Q6_K:
        w[:, :192] = np.where(np.arange(w.shape[0])[:, None] % 2, 0xFF, 0x00)   # 31 or -32 ...
        w[:, 192:208] = 0x80                                                    # ... times -128
        w[:, 208:210] = np.frombuffer(np.float16(0.01).tobytes(), dtype=np.uint8)
    xs = np.ones(m * cols, dtype=np.float32)
    xs[cols:2 * cols] = -1.0                          # every quant -127, or 127
    _run(pkg, ob, ctx, kind, w.reshape(-1), xs, m, rows, cols, f"kind {kind} at the bounds")


@pytest.fixture
def cluster_kernel(pkg, ctx):
    """K-quant batches on the tcgen05 kernel of clusters whatever their size."""
    spec = pkg.model.tiny("llama", n_layer=1)
    g = pkg.Gpu(ctx, spec.head, spec.layers, spec.weights, 16, 2)
    g.set_option("k_tensor", 2)
    g.set_option("wide_multi", 0)
    yield g
    for name, value in (("k_tensor", 0), ("wide_multi", 1), ("kt_cluster", 0)):
        g.set_option(name, value)
    g.close()


# Which of the two batch kernels is taken: measured, one is 10 % to twice as fast.
@pytest.mark.parametrize("kind,rows,cols,m,cluster", [(Q6_K, 5632, 2048, 8, False), (Q6_K, 2048, 256, 40, False), (Q5_K, 1024, 1024, 48, False), (Q4_K, 300, 14336, 4, False),
                                                      (Q6_K, 2049, 5632, 48, False), (Q4_K, 24576, 4096, 64, True), (Q5_K, 4096, 14336, 64, True), (Q6_K, 4096, 14336, 64, True)])
def test_k_quant_choice_of_kernel(pkg, ob, ctx, kind, rows, cols, m, cluster):
    spec = pkg.model.tiny("llama", n_layer=1)
    g = pkg.Gpu(ctx, spec.head, spec.layers, spec.weights, 16, 2)
    before = _launches(g)[0]
    _run(pkg, ob, ctx, kind, make_weights(pkg, kind, rows, cols, 39 + kind, "uniform"), np.random.default_rng(m).standard_normal(m * cols).astype(np.float32), m, rows, cols,
         f"kind {kind} {rows}x{cols} m {m}")
    assert _launches(g)[0] - before == int(cluster)
    g.close()


# Fewer super-blocks than CTAs in a cluster, a last stage with some of them, rows that tensor copies
# cannot take (Q6_K: 768 and 2304 columns), a partial row tile, several tiles per cluster, token groups
# of every parity and a second launch.
@pytest.mark.parametrize("kind", [Q4_K, Q5_K, Q6_K])
@pytest.mark.parametrize("cluster", [2, 4, 8])
def test_k_quant_clusters(pkg, ob, ctx, cluster_kernel, kind, cluster):
    cluster_kernel.set_option("kt_cluster", cluster)
    for rows, cols, ms in ((1, 256, (2, 64)), (129, 2048, (8, 17, 33, 48)), (300, 768, (25, 65)), (9700, 2304, (64,))):
        w = make_weights(pkg, kind, rows, cols, 25 + kind + rows, "uniform")
        for m in ms:
            before = _launches(cluster_kernel)[0]
            _run(pkg, ob, ctx, kind, w, np.random.default_rng(m).standard_normal(m * cols).astype(np.float32), m, rows, cols, f"kind {kind} {rows}x{cols} m {m} clusters of {cluster}")
            assert _launches(cluster_kernel)[0] - before == (m + 63) // 64


@pytest.mark.parametrize("kind", [Q4_K, Q6_K])
def test_k_quant_clusters_pairs_bounds_and_offsets(pkg, ob, ctx, cluster_kernel, kind):
    rows, cols, m = 70, 2048, 40                       # a pair: 64 rows of each per tile
    ws = [make_weights(pkg, kind, rows, cols, 27 + i, "uniform") for i in range(2)]
    b = ws[0].reshape(rows * cols // 256, -1)
    if kind == Q6_K:                                   # quants 31 or -32 times -128, and the largest of Q4_K
        b[:, :192], b[:, 192:208] = np.where(np.arange(b.shape[0])[:, None] % 2, 0xFF, 0x00), 0x80
    else:
        b[:, 4:] = 0xFF
    xs = np.random.default_rng(m).standard_normal(m * cols).astype(np.float32)
    xs[:cols], xs[cols:2 * cols] = 1.0, -1.0
    q = ob.quantize_act(kind, xs)
    dq, outs = ctx.to_device(q.view(np.uint8)), [ctx.alloc(m * rows * 4) for _ in ws]
    want = [ob.matmul(ob.Pool(4), ob.detect_table(), kind, w, q, m, rows, cols) for w in ws]
    before = _launches(cluster_kernel)[0]
    ctx.matmul2(kind, *outs, *[ctx.to_device(w) for w in ws], dq, m, rows, cols)
    for o, x in zip(outs, want):
        assert_bits_equal(o.download(np.float32, m * rows).reshape(m, rows), x, "pair")
    off = 2 if kind == Q6_K else 16                    # a base that tensor copies cannot take, or can
    d = ctx.to_device(np.concatenate([np.zeros(off, np.uint8), ws[0].reshape(-1), np.zeros(256, np.uint8)]))
    ctx.matmul(kind, outs[0], d.ptr + off, dq, m, rows, cols)
    assert_bits_equal(outs[0].download(np.float32, m * rows).reshape(m, rows), want[0], f"offset {off}")
    assert _launches(cluster_kernel)[0] - before == 2
    ctx.device_status()


# What follows a wait that runs out: the kernel ends, the status says so, and the next product is right. No CTA may wait
# for one that has left: every CTA of a cluster makes that many requests, before it needs anything of its peers.
# Copied by tensor copies or not (Q6_K, 768 columns), one stage per tile, several; pairs, whose warps meet at every tile.
@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("kind,cluster,cols,after", [(Q4_K, 4, 1024, 1), (Q4_K, 4, 1024, 2), (Q4_K, 2, 1024, 3), (Q6_K, 8, 2048, 2), (Q6_K, 2, 768, 1)])
def test_k_quant_clusters_after_a_wait_that_gave_up(pkg, ob, ctx, cluster_kernel, kind, cluster, cols, after, pair):
    cluster_kernel.set_option("kt_cluster", cluster)
    rows, m = 3 * 148 * 128, 40                        # at least three tiles per cluster
    dw, dout, dout2 = ctx.alloc(rows * cols // 256 * (144 if kind == Q4_K else 210)), ctx.alloc(m * rows * 4), ctx.alloc(m * rows * 4)
    dq = ctx.to_device(ob.quantize_act(kind, np.ones(m * cols, np.float32)).view(np.uint8))
    before = _launches(cluster_kernel)[0]
    cluster_kernel.set_option("give_up", after)
    try:
        if pair:
            ctx.matmul2(kind, dout, dout2, dw, dw, dq, m, rows, cols)
        else:
            ctx.matmul(kind, dout, dw, dq, m, rows, cols)
        with pytest.raises(pkg.AotCudaError, match="wait expired"):
            ctx.device_status()
    finally:
        cluster_kernel.set_option("give_up", 0)
    w = make_weights(pkg, kind, 129, cols, 35 + kind, "uniform")
    _run(pkg, ob, ctx, kind, w, np.random.default_rng(m).standard_normal(m * cols).astype(np.float32), m, 129, cols, f"kind {kind} after a wait that gave up")
    assert _launches(cluster_kernel)[0] - before == 2


@pytest.mark.parametrize("kind", [Q4_K, Q6_K])
def test_k_quant_batch_where_one_order_of_the_activations_fits(pkg, ob, ctx, cluster_kernel, kind):
    """8 token groups x 56 super-blocks: 448 blocks of 2336 bytes (mma.sync kernel) are below 1 MiB, of 2368 (clusters)
    above it. A conversion and a product all the same, not the per-token kernel."""
    rows, cols, m = 130, 56 * 256, 64
    w = make_weights(pkg, kind, rows, cols, 29 + kind, "uniform")
    cluster_kernel.set_option("workspace_mib", 0)      # gives back a larger buffer
    cluster_kernel.set_option("workspace_mib", 1)
    before, kt = cluster_kernel.dispatches(), _launches(cluster_kernel)[0]
    try:
        _run(pkg, ob, ctx, kind, w, np.random.default_rng(m).standard_normal(m * cols).astype(np.float32), m, rows, cols, f"kind {kind} under a bound")
    finally:
        cluster_kernel.set_option("workspace_mib", 1 << 20)
    assert cluster_kernel.dispatches() - before == 2 and _launches(cluster_kernel)[0] == kt


def test_k_quant_clusters_in_a_model(pkg, ob, ctx, cluster_kernel):
    """q/k/v of mixed kinds, gated pairs and products onto the residual, chunk after chunk."""
    spec = pkg.model.tiny("llama", n_layer=2, kinds=lambda layer, tensor: Q6_K if tensor in ("wv", "down", "output") else Q4_K, dim=512, hidden=768, vocab=600)
    g = pkg.Gpu(ctx, spec.head, spec.layers, spec.weights, 160, 64)
    om = ob.model_from_spec(spec, 160, 64, n_threads=4)
    pos = 0
    for n in (64, 21, 9, 8):
        before = _launches(g)[0]
        toks = np.random.default_rng(n).integers(0, 600, n).tolist()
        g.forward_batch(toks, pos, True)
        om.forward_batch(toks, pos, True)
        assert_bits_equal(g.logits(), om.logits(), f"logits after a chunk of {n} at {pos}")
        # per layer q/k of one kind and v of another, wo, gate/up, down; up to eight rows lie in the other kernel's order only
        assert _launches(g)[0] - before == (10 if n > 8 else 0)
        pos += n
    g.close()
    ctx.device_status()


@pytest.mark.parametrize("kind", [0, 1, 2])           # F32, F16, BF16
@pytest.mark.parametrize("rows,cols", [(1, 8), (33, 72), (600, 1016), (5000, 128)])
def test_float_tile_edges(pkg, ob, ctx, kind, rows, cols):
    w = make_weights(pkg, kind, rows, cols, 31 + kind + rows)
    for m in (2, 3, 5, 9, 41, 64):                    # 41: a last warp with one row, two CTAs per row tile
        xs = np.random.default_rng(m).standard_normal(m * cols).astype(np.float32)
        _run(pkg, ob, ctx, kind, w, xs, m, rows, cols, f"kind {kind} {rows}x{cols} m {m}")


# Batches for which the streaming kernel's estimate is the lower one, in each of its forms: rows of a
# CTA in one or two quads per lane, two token groups of eight with four rows per lane (or, by option,
# sixteen tokens per lane), up to eight tokens, pairs; 28 rows are two launches of it.
@pytest.mark.parametrize("kind,rows,pair,ms", [(1, 5632, False, (13,)), (2, 14336, False, (8, 16, 28)), (0, 2560, False, (9, 14)),
                                               (0, 11264, False, (16,)), (1, 4096, True, (16,)), (2, 5632, True, (7, 15)), (0, 5632, True, (13,))])
def test_float_batches_on_the_streaming_kernel(pkg, ob, ctx, kind, rows, pair, ms):
    cols = 520
    spec = pkg.model.tiny("llama", n_layer=1)
    g = pkg.Gpu(ctx, spec.head, spec.layers, spec.weights, 16, 2)  # for the option and the count of launches
    ws = [make_weights(pkg, kind, rows, cols, 33 + i) for i in range(1 + pair)]
    dws = [ctx.to_device(w) for w in ws]
    try:
        for rows4 in (0, 1):
            g.set_option("float_rows4", rows4)
            for m in ms:
                x = np.random.default_rng(m).standard_normal(m * cols).astype(np.float32)
                dx, outs = ctx.to_device(x), [ctx.alloc(m * rows * 4) for _ in ws]
                before = g.dispatches()
                if pair:
                    ctx.matmul2(kind, *outs, *dws, dx, m, rows, cols)
                else:
                    ctx.matmul(kind, outs[0], dws[0], dx, m, rows, cols)
                assert g.dispatches() - before == (m + 15) // 16
                for o, w in zip(outs, ws):
                    assert_bits_equal(o.download(np.float32, m * rows).reshape(m, rows), ob.matmul(ob.Pool(4), ob.detect_table(), kind, w, x, m, rows, cols),
                                      f"kind {kind} {rows}x{cols} m {m} rows4 {rows4}")
    finally:
        g.set_option("float_rows4", 1)
        g.close()
    ctx.device_status()


@pytest.mark.parametrize("kind", [3, 4, 5])           # Q4_0, Q5_0, Q8_0
def test_q80_tile_edges(pkg, ob, ctx, batch_kernels, kind):
    for rows, cols, ms in ((8192, 256, (49, 64)), (8205, 768, (50, 81, 129))):   # a partial row tile, half-full warps, two CTAs per tile
        w = make_weights(pkg, kind, rows, cols, 41 + kind)
        for m in ms:
            xs = np.random.default_rng(m).standard_normal(m * cols).astype(np.float32)
            _run(pkg, ob, ctx, kind, w, xs, m, rows, cols, f"kind {kind} {rows}x{cols} m {m}")


# Both sides of the choice between the streaming and the matrix-instruction kernel: few rows and
# many tokens, two and three warps per CTA, five with one CTA per SM, rows not in fours; and products
# just before it.
@pytest.mark.parametrize("kind,rows,cols,m,mma", [(3, 300, 512, 128, True), (4, 260, 256, 112, True), (5, 4100, 512, 81, True), (3, 11264, 256, 32, True),
                                                  (5, 8192, 256, 48, True), (4, 12000, 512, 17, True), (3, 16400, 256, 80, True),
                                                  (3, 301, 512, 32, True), (3, 300, 512, 32, False), (5, 2048, 512, 48, False), (4, 8192, 256, 16, False)])
def test_q80_sizes_around_the_choice_of_kernel(pkg, ob, ctx, kind, rows, cols, m, mma):
    """On the kernels of warp-level instructions alone, whose choice this is; then as products get them."""
    spec = pkg.model.tiny("llama", n_layer=1)
    g = pkg.Gpu(ctx, spec.head, spec.layers, spec.weights, 16, 2)  # for the count of launches
    w = make_weights(pkg, kind, rows, cols, 43 + kind)
    xs = np.random.default_rng(m).standard_normal(m * cols).astype(np.float32)
    qt = _launches(g)[1]
    g.set_option("q80_tensor", 1)
    before = g.dispatches()
    try:
        _run(pkg, ob, ctx, kind, w, xs, m, rows, cols, f"kind {kind} {rows}x{cols} m {m}")
    finally:
        g.set_option("q80_tensor", 0)
    assert g.dispatches() - before == (2 if mma else 1 + (m + 15) // 16)
    assert _launches(g)[1] == qt
    before = g.dispatches()
    _run(pkg, ob, ctx, kind, w, xs, m, rows, cols, f"kind {kind} {rows}x{cols} m {m} by estimates")
    assert g.dispatches() - before == (2 if mma or _launches(g)[1] != qt else 1 + (m + 15) // 16)
    g.close()


@pytest.fixture
def q80_tensor(pkg, ctx):
    """Q8_0-family batches on the tcgen05 kernel whatever their size."""
    spec = pkg.model.tiny("llama", n_layer=1)
    g = pkg.Gpu(ctx, spec.head, spec.layers, spec.weights, 16, 2)
    g.set_option("q80_tensor", 2)
    yield g
    g.set_option("q80_tensor", 0)
    g.set_option("q80_tensor_rows", 0)
    g.close()


# One row, a partial row tile, several tiles per CTA, one to three stages; every number of tokens per CTA
# with a partial group; pairs; all products of one sign with zeros, whose sums must not become -0.
@pytest.mark.parametrize("kind", [3, 4, 5])           # Q4_0, Q5_0, Q8_0
@pytest.mark.parametrize("tokens", [16, 24, 32])
def test_q80_on_tcgen05(pkg, ob, ctx, q80_tensor, kind, tokens):
    q80_tensor.set_option("q80_tensor_rows", tokens)
    before = _launches(q80_tensor)[1]
    for rows, cols, ms in ((1, 256, (2, 65)), (301, 768, (17, 33, 64)), (19100, 256, (40,))):
        w = make_weights(pkg, kind, rows, cols, 45 + kind + rows)
        for m in ms:
            _run(pkg, ob, ctx, kind, w, np.random.default_rng(m).standard_normal(m * cols).astype(np.float32), m, rows, cols, f"kind {kind} {rows}x{cols} m {m}, {tokens} per CTA")
    rows, cols, m = 70, 512, 37
    ws = [make_weights(pkg, kind, rows, cols, 53 + i) for i in range(2)]
    b = ws[1].reshape(rows * cols // 32, -1)
    b[:, 2:] = 0x80 if kind == 5 else 0x00            # the lowest quants
    xs = np.random.default_rng(m).standard_normal(m * cols).astype(np.float32)
    xs[:cols] = 0.0
    q = ob.quantize_act(kind, xs)
    outs = [ctx.alloc(m * rows * 4) for _ in ws]
    ctx.matmul2(kind, *outs, *[ctx.to_device(w) for w in ws], ctx.to_device(q.view(np.uint8)), m, rows, cols)
    for o, w in zip(outs, ws):
        assert_bits_equal(o.download(np.float32, m * rows).reshape(m, rows), ob.matmul(ob.Pool(4), ob.detect_table(), kind, w, q, m, rows, cols), "pair")
    assert _launches(q80_tensor)[1] - before == 7
    ctx.device_status()


@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("kind,after", [(3, 1), (4, 3), (5, 6)])
def test_q80_on_tcgen05_after_a_wait_that_gave_up(pkg, ob, ctx, q80_tensor, kind, after, pair):
    rows, cols, m = 2 * 148 * 128, 1024, 40
    dw, dout, dout2 = ctx.alloc(rows * cols // 32 * {3: 18, 4: 22, 5: 34}[kind]), ctx.alloc(m * rows * 4), ctx.alloc(m * rows * 4)
    dq = ctx.to_device(ob.quantize_act(kind, np.ones(m * cols, np.float32)).view(np.uint8))
    before = _launches(q80_tensor)[1]
    q80_tensor.set_option("give_up", after)
    try:
        if pair:
            ctx.matmul2(kind, dout, dout2, dw, dw, dq, m, rows, cols)
        else:
            ctx.matmul(kind, dout, dw, dq, m, rows, cols)
        with pytest.raises(pkg.AotCudaError, match="wait expired"):
            ctx.device_status()
    finally:
        q80_tensor.set_option("give_up", 0)
    w = make_weights(pkg, kind, 129, cols, 37 + kind)
    _run(pkg, ob, ctx, kind, w, np.random.default_rng(m).standard_normal(m * cols).astype(np.float32), m, 129, cols, f"kind {kind} after a wait that gave up")
    assert _launches(q80_tensor)[1] - before == 2


def test_q80_on_tcgen05_in_a_model(pkg, ob, ctx, q80_tensor):
    """Gated pairs and products onto the residual, chunk after chunk."""
    spec = pkg.model.tiny("llama", n_layer=2, kinds=lambda layer, tensor: 3 if tensor in ("gate", "up", "wq") else 5, dim=512, hidden=768, vocab=600)
    g = pkg.Gpu(ctx, spec.head, spec.layers, spec.weights, 160, 64)
    om = ob.model_from_spec(spec, 160, 64, n_threads=4)
    pos = 0
    before = _launches(g)[1]
    for n in (64, 21, 9):
        toks = np.random.default_rng(n).integers(0, 600, n).tolist()
        g.forward_batch(toks, pos, True)
        om.forward_batch(toks, pos, True)
        assert_bits_equal(g.logits(), om.logits(), f"logits after a chunk of {n} at {pos}")
        pos += n
    assert _launches(g)[1] - before == 3 * 10          # per layer wq, wk and wv, wo, gate/up, down
    g.close()
    ctx.device_status()


@pytest.mark.parametrize("kind,rows,cols", [(0, 20, 64), (1, 37, 20), (3, 301, 256), (5, 64, 96), (6, 40, 256), (8, 3, 512)])
def test_batches_longer_than_a_pass(pkg, ob, ctx, kind, rows, cols):
    m = 4096 + 9 if cols % 32 == 0 else 8192 + 3
    w = make_weights(pkg, kind, rows, cols, 47 + kind)
    _run(pkg, ob, ctx, kind, w, np.random.default_rng(kind).standard_normal(m * cols).astype(np.float32), m, rows, cols, f"kind {kind} {rows}x{cols} m {m}")


def test_q80_pair_tile_edges(pkg, ob, ctx, batch_kernels):
    rows, cols, m = 4105, 512, 60
    ws = [make_weights(pkg, 3, rows, cols, 51 + i) for i in range(2)]
    q = ob.quantize_act(3, np.random.default_rng(m).standard_normal(m * cols).astype(np.float32))
    outs = [ctx.alloc(m * rows * 4) for _ in ws]
    ctx.matmul2(3, *outs, *[ctx.to_device(w) for w in ws], ctx.to_device(q.view(np.uint8)), m, rows, cols)
    for o, w in zip(outs, ws):
        assert_bits_equal(o.download(np.float32, m * rows).reshape(m, rows), ob.matmul(ob.Pool(4), ob.detect_table(), 3, w, q, m, rows, cols), "pair")
    ctx.device_status()
