"""Attention at the sizes where its kernel changes path: query groups that span rows and are not
full, head widths that are not whole pieces, windows, more positions than the scores' shared
memory holds. Bit-exact against the CPU oracle (crates/aot-kernels/src/ops.rs:517-556)."""
import numpy as np
import pytest

from conftest import assert_bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_head,n_kv,hd,ctxlen,calls", [
    (6, 2, 20, 700, [(1, 699, 0), (11, 600, 0), (64, 300, 77)]),     # three heads per group, a partial piece
    (1, 1, 256, 300, [(1, 0, 0), (9, 290, 33)]),                      # one query per row, widest heads
    (24, 2, 64, 260, [(3, 0, 0), (5, 255, 0)]),                       # twelve heads per group: two CTAs a row
    (4, 1, 32, 6200, [(1, 6100, 0), (3, 6190, 0), (2, 6000, 5900)]),  # few CTAs: four queries each
    (4, 1, 32, 12000, [(3, 11990, 0)]),                               # the same, scores in global memory
    (32, 4, 16, 6200, [(64, 6130, 0), (40, 6100, 3000)]),             # eight queries each, scores in global memory
])
def test_attention_paths(pkg, ob, ctx, n_head, n_kv, hd, ctxlen, calls):
    rng = np.random.default_rng(hd)
    kc, vc = (rng.standard_normal(ctxlen * n_kv * hd).astype(np.float32) for _ in range(2))
    d = ob.Dims()
    d.n_head, d.n_kv_head, d.head_dim = n_head, n_kv, hd
    dk, dv = ctx.to_device(kc), ctx.to_device(vc)
    for m, pos0, window in calls:
        q = rng.standard_normal(m * n_head * hd).astype(np.float32)
        dout = ctx.alloc(q.nbytes)
        ctx.attention(dout, ctx.to_device(q), dk, dv, n_head, n_kv, hd, ctxlen, pos0, m, window)
        assert_bits_equal(dout.download(np.float32, q.size), ob.attention_rows(ob.Pool(4), q, kc, vc, d, ctxlen, 0, pos0, m, window),
                          f"m {m} pos0 {pos0} window {window}")
    ctx.device_status()


def test_misaligned_caches_are_refused(pkg, ctx):
    hd, n = 32, 8
    dq, dk, dv = ctx.alloc(hd * 4), ctx.alloc((n + 1) * hd * 4), ctx.alloc((n + 1) * hd * 4)
    for k, v in ((dk.at(4), dv), (dk, dv.at(8))):
        with pytest.raises(pkg.AotCudaError) as e:
            ctx.attention(dq, dq, k, v, 1, 1, hd, n, 0, 1, 0)
        assert e.value.status == pkg.lib.ERR_BAD_ARG
    ctx.device_status()


# Heads whose outputs make whole blocks of 256 in a CTA of four or eight queries (one or two rows of a
# group of heads), heads that do not, and 32-value blocks; few rows and many.
@pytest.mark.parametrize("kind", [5, 6])              # Q8_0, Q4_K
@pytest.mark.parametrize("n_head,n_kv,head_dim", [(8, 2, 64), (8, 1, 64), (4, 1, 128), (2, 2, 128), (8, 2, 32), (1, 1, 256)])
def test_attention_output_quantized_on_the_way(pkg, ob, ctx, kind, n_head, n_kv, head_dim):
    spec = pkg.model.build("attn", dim=512, hidden=512, n_layer=2, n_head=n_head, n_kv_head=n_kv, head_dim=head_dim, vocab=300, seed=5,
                           kinds=lambda layer, tensor: 6 if tensor in ("token_embd", "output") else kind, n_ctx_train=512, rope_base=1e4, eps=1e-5)
    g, om = pkg.Gpu(ctx, spec.head, spec.layers, spec.weights, 96, 64), ob.model_from_spec(spec, 96, 64, n_threads=4)
    pos = 0
    for n in (64, 3, 9):
        toks = np.random.default_rng(n).integers(0, 300, n).tolist()
        g.forward_batch(toks, pos, True)
        om.forward_batch(toks, pos, True)
        assert_bits_equal(g.logits(), om.logits(), f"logits after a chunk of {n} at {pos}")
        pos += n
    g.close()
    ctx.device_status()
