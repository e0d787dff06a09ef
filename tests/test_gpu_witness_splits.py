"""Witness products where the kernels' forms change: one, two and four CTAs of a cluster on a column tile and several clusters, result
rows that take 32-byte, 16-byte and single stores, and weights that are copied with every alignment of their rows, both layouts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from intelligenceregulation_b200 import backend

    c = backend.Context(0)
    yield c
    c.close()


CASES = [(128, 128 * k, n, n, False) for k, n in ((1, 256), (2, 256), (3, 512), (17, 600), (9, 20000))]  # stages against splits
CASES += [(3, 256, n, os_, False) for n, os_ in ((260, 260), (258, 258), (257, 257), (256, 259), (260, 262))]  # stores
CASES += [(2, k, n, n, lay) for k, n in ((127, 129), (130, 131), (255, 126), (129, 4), (3, 385)) for lay in (False, True)]  # copies


@pytest.mark.parametrize("t,k,n,os_,in_out", CASES)
def test_product(ctx, oracle, t, k, n, os_, in_out):
    rng = np.random.default_rng(t + 3 * k + 5 * n)
    x = rng.integers(-32768, 32768, size=t * k, dtype=np.int64)
    w = rng.integers(-128, 128, size=k * n, dtype=np.int8)
    want = oracle.witness_product(t, x, k, w, k, n, os_, t * os_, in_out)
    got = ctx.witness_product(t, x, k, w, k, n, os_, t * os_, in_out)
    assert got is not None and (got == want).all()
