"""Operator calls on parts of a buffer: offsets and row lengths that the step itself never uses.
Bit-exact against the CPU oracle (batched == per-token, crates/aot-kernels/tests/dots.rs:205-266)."""
import numpy as np
import pytest

from conftest import assert_bits_equal, make_weights

pytestmark = pytest.mark.gpu

KINDS = [0, 1, 5, 6, 8]  # F32, F16, Q8_0, Q4_K, Q6_K


def _model_with(pkg, ctx, mats, n_ctx, max_batch):
    """A small model whose tensor section also holds `mats` ((kind, rows, cols) each)."""
    spec = pkg.model.tiny("llama", n_layer=1)
    parts, off, out = [spec.weights], spec.weights.size, []
    for kind, rows, cols in mats:
        w = make_weights(pkg, kind, rows, cols, 61 + kind + cols)
        pad = -off % 32
        parts += [np.zeros(pad, dtype=np.uint8), w]
        out.append((w, pkg.lib.Tensor(kind=kind, present=1, off=off + pad, len=w.size, rows=rows, cols=cols)))
        off += pad + w.size
    return pkg.Gpu(ctx, spec.head, spec.layers, np.concatenate(parts), n_ctx, max_batch), out


def _want(ob, kind, w, x, m, rows, cols):
    return ob.matmul(ob.Pool(4), ob.detect_table(), kind, w, ob.quantize_act(kind, x), m, rows, cols)


@pytest.mark.parametrize("src_off,dst_off", [(0, 0), (1, 3), (2, 0), (4, 1)])
def test_matmul_of_a_part_of_a_buffer(pkg, ob, ctx, src_off, dst_off):
    rows, cols = 48, 512
    g, mats = _model_with(pkg, ctx, [(k, rows, cols) for k in KINDS], 16, 16)
    for (w, t), kind in zip(mats, KINDS):
        for m in (1, 2, 9):
            x = np.random.default_rng(kind + m).standard_normal(m * cols).astype(np.float32)
            g.write("Bhb", x, src_off)
            g.matmul("Bq", t, "Bhb", m, src_off=src_off, dst_off=dst_off)
            assert_bits_equal(g.read("Bq", m * rows, dst_off).reshape(m, rows), _want(ob, kind, w, x, m, rows, cols), f"kind {kind} m {m} at {src_off}")
    g.finish()
    g.close()


def test_rows_longer_than_any_of_the_model(pkg, ob, ctx):
    """Quantized rows that do not fit the activation buffer in groups of eight, or not at all."""
    cases = [(6, 48, 4096, 2), (8, 2800, 2560, 3), (6, 48, 768, 9), (5, 48, 4096, 2)]
    too_long = [(6, 4, 16384), (5, 4, 16384)]
    g, mats = _model_with(pkg, ctx, [c[:3] for c in cases] + too_long, 256, 16)
    for (kind, rows, cols, m), (w, t) in zip(cases, mats):
        x = np.random.default_rng(cols).standard_normal(m * cols).astype(np.float32)
        g.write("Bhb", x)
        g.matmul("KCache", t, "Bhb", m)
        assert_bits_equal(g.read("KCache", m * rows).reshape(m, rows), _want(ob, kind, w, x, m, rows, cols), f"kind {kind} {rows}x{cols} m {m}")
    for _, t in mats[len(cases):]:
        with pytest.raises(pkg.AotCudaError) as e:
            g.matmul("Q", t, "KCache")
        assert e.value.status == pkg.lib.ERR_BAD_ARG
    # a norm of such a row is computed, and not quantized
    n = 16384
    g2, [(w, t)] = _model_with(pkg, ctx, [(0, 1, n)], 256, 16)
    x = np.random.default_rng(3).standard_normal(n).astype(np.float32)
    g2.write("KCache", x)
    g2.rmsnorm("VCache", "KCache", t, n, 1, 1e-5)
    assert_bits_equal(g2.read("VCache", n), ob.rmsnorm(x, w.view(np.float32), 1e-5), "norm of a long row")
    for h in (g, g2):
        h.finish()
        h.close()


@pytest.mark.parametrize("kind,rows,cols,ms", [(3, 8192, 256, (2, 64)), (4, 600, 1024, (17,)), (5, 8200, 512, (49,)),
                                               (6, 2400, 512, (4, 65)), (7, 900, 1280, (12,)), (8, 2400, 768, (9,))])
def test_products_without_a_conversion_buffer(pkg, ob, ctx, kind, rows, cols, ms):
    """What a product does when the buffer for its activations cannot be had."""
    g, _ = _model_with(pkg, ctx, [], 16, 2)  # only to reach the context's option
    ws = [make_weights(pkg, kind, rows, cols, 71 + kind + i) for i in range(2)]
    dws = [ctx.to_device(w) for w in ws]
    try:
        for limit in (0, 1 << 20):  # 1 << 20 MiB: as good as none
            g.set_option("workspace_mib", limit)
            for m in ms:
                x = np.random.default_rng(m).standard_normal(m * cols).astype(np.float32)
                q = ob.quantize_act(kind, x)
                dq = ctx.to_device(q.view(np.uint8))
                want = [ob.matmul(ob.Pool(4), ob.detect_table(), kind, w, q, m, rows, cols) for w in ws]
                outs = [ctx.alloc(m * rows * 4) for _ in ws]
                ctx.matmul(kind, outs[0], dws[0], dq, m, rows, cols)
                assert_bits_equal(outs[0].download(np.float32, m * rows).reshape(m, rows), want[0], f"kind {kind} m {m} limit {limit}")
                ctx.matmul2(kind, *outs, *dws, dq, m, rows, cols)
                for i in range(2):
                    assert_bits_equal(outs[i].download(np.float32, m * rows).reshape(m, rows), want[i], f"pair, kind {kind} m {m} limit {limit}")
    finally:
        g.set_option("workspace_mib", 1 << 20)
        g.close()
    ctx.device_status()


def test_a_write_inside_a_quantized_row_is_seen(pkg, ob, ctx):
    rows, cols, m = 48, 512, 2
    g, mats = _model_with(pkg, ctx, [(k, rows, cols) for k in (5, 6)], 16, 16)
    for (w, t), kind in zip(mats, (5, 6)):
        x = np.random.default_rng(kind).standard_normal(m * cols).astype(np.float32)
        g.write("Bhb", x)
        g.matmul("Bq", t, "Bhb", m)
        x[700:720] = 3.0
        g.write("Bhb", x[700:720], 700)
        g.matmul("Bq", t, "Bhb", m)
        assert_bits_equal(g.read("Bq", m * rows).reshape(m, rows), _want(ob, kind, w, x, m, rows, cols), f"kind {kind}")
    g.finish()
    g.close()
