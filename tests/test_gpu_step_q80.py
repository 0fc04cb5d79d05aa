"""The one-kernel decode step on models whose layers are of the Q8_0 family: kinds mixed inside a
phase (a warp's four rows may be of two kinds), row shares that are not multiples of four, K-quant
and Q8_0-family output heads, contexts that one CTA per head no longer holds. Bit-exact against the
CPU oracle and the per-operator path."""
import numpy as np
import pytest

from conftest import assert_bits_equal

pytestmark = pytest.mark.gpu

Q4_0, Q5_0, Q8_0, Q6_K = 3, 4, 5, 8


@pytest.mark.parametrize("arch,head,shape", [
    ("llama", Q6_K, dict(dim=512, hidden=768, vocab=600)),
    ("qwen3", Q8_0, dict(dim=256, hidden=2048, vocab=333)),
])
def test_q80_step_bit_exact(pkg, ob, ctx, arch, head, shape):
    def kinds(layer, tensor):
        if tensor == "output":
            return head
        name = "gate" if tensor == "up" else tensor
        return [Q4_0, Q5_0, Q8_0][(layer + len(name) + ord(name[-1])) % 3]

    n_ctx = 1100
    spec = pkg.model.tiny(arch, n_layer=3, kinds=kinds, **shape)
    g = pkg.Gpu(ctx, spec.head, spec.layers, spec.weights, n_ctx, 64)
    assert g.set_option("mega_available", 0)
    tokens = np.random.default_rng(3).integers(0, shape["vocab"], n_ctx)
    for mega in (1, 0):
        g.set_option("mega", mega)
        om = ob.model_from_spec(spec, n_ctx, 64, n_threads=4)
        for pos in range(6):
            g.forward(int(tokens[pos]), pos, True)
            om.forward(int(tokens[pos]), pos, True)
            assert_bits_equal(g.read("X"), om.buf("x"), f"x pos {pos} mega {mega}")
            assert_bits_equal(g.logits(), om.logits(), f"logits pos {pos} mega {mega}")
    want = None
    for mega in (1, 0):                                # long contexts: the two paths against one another
        g.set_option("mega", mega)
        for a in range(0, 1024, 64):
            g.forward_batch(tokens[a:a + 64], a, False)
        ids, _ = g.generate(int(tokens[1024]), 1024, 8)
        got = (ids.tolist(), g.logits().view(np.uint32).tolist())
        want = want or got
        assert got == want
    ctx.device_status()
