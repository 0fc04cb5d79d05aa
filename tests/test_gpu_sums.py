"""The sequential f32 sum of squares of rmsnorm (crates/aot-kernels/src/ops.rs:7-18), evaluated in
parallel, on rows that send it down each of its paths: a plain chain, one and several rounds of
groups, exact ties, more binades than a round holds, sums too small for its integer steps, and
predictions that meet a sum on a binade boundary. Bit-exact against the CPU oracle."""
import numpy as np
import pytest

from conftest import assert_bits_equal

pytestmark = pytest.mark.gpu


def _rows(n, rng):
    normal = rng.standard_normal(n)
    outlier = normal.copy()
    outlier[n // 3] = 3e4
    return {
        "normal": normal, "outlier": outlier, "growing": 2.0 ** (np.arange(n) * 30.0 / n) * normal,
        "tiny": normal * 1e-18, "subnormal squares": normal * 1e-21, "ties": rng.integers(0, 3, n) * 0.5,
        "boundary": np.full(n, 0.5), "zeros": np.where(np.arange(n) < n - 2, 0.0, 1.0), "huge": normal * 1e17,
    }


@pytest.mark.parametrize("n", [768, 769, 2048, 2051, 4096, 4100, 8448])
def test_rmsnorm_sum_paths(pkg, ob, ctx, n):
    rng = np.random.default_rng(n)
    w = (1 + rng.random(n)).astype(np.float32)
    rows = {k: v.astype(np.float32) for k, v in _rows(n, rng).items()}
    x = np.concatenate(list(rows.values()))
    dout = ctx.alloc(x.nbytes)
    ctx.rmsnorm(dout, ctx.to_device(x), ctx.to_device(w), n, len(rows), 1e-5)
    got = dout.download(np.float32, x.size).reshape(len(rows), n)
    for (name, row), g in zip(rows.items(), got):
        assert_bits_equal(g, ob.rmsnorm(row, w, 1e-5), f"n {n}: {name}")
    ctx.device_status()
