"""Field read-back through the pipelined copy (csrc/engine.cu, copy_out): the
values written come back unchanged, below and above the size where it starts,
with padded rows, on 2-byte storage, from several threads at once."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

import openems_b200 as oe

pytestmark = pytest.mark.gpu


def engine(dims, **kw):
    return oe.Engine(oe.Operator(oe.Grid.uniform(*dims, 1e-3), oe.BoundaryConditions.all_pec()), **kw)


# 24 B a cell against 1 MB: below; just above; rows padded by 1-3; pieces of
# the full 4 MB; one row longer than a piece
@pytest.mark.parametrize("dims", [(20, 30, 41), (36, 35, 37), (70, 71, 72), (150, 140, 143), (80, 81, 83), (64, 100, 129), (1, 2, 1100001)])
def test_fields_come_back(dims):
    eng = engine(dims)
    rng = np.random.default_rng(3)
    f = rng.standard_normal((2, 3) + dims, dtype=np.float32)
    eng.write_fields(f[0], f[1])
    for _ in range(2):
        e, h = eng.read_fields()
        assert np.array_equal(e, f[0]) and np.array_equal(h, f[1])


@pytest.mark.parametrize("storage,bits", [("f16", 11), ("bf16", 8)])
@pytest.mark.parametrize("dims", [(9, 10, 11), (90, 91, 93)])
def test_two_byte_storage(storage, bits, dims):
    """Values of at most `bits` significant bits survive the storage exactly."""
    eng = engine(dims, storage=storage)
    rng = np.random.default_rng(4)
    f = rng.integers(-(1 << bits) + 1, 1 << bits, (2, 3) + dims).astype(np.float32) / 4096
    f[1] /= 64
    eng.write_fields(f[0], f[1])
    e, h = eng.read_fields()
    assert np.array_equal(e, f[0]) and np.array_equal(h, f[1])


def test_several_threads():
    engs = [engine((60 + k, 80, 90)) for k in range(4)]
    fields = [np.random.default_rng(k).standard_normal((2, 3) + tuple(e.dims), dtype=np.float32)
              for k, e in enumerate(engs)]
    for e, f in zip(engs, fields):
        e.write_fields(f[0], f[1])
    with ThreadPoolExecutor(4) as pool:
        for got, f in zip(pool.map(lambda e: np.stack(e.read_fields()), engs * 3), fields * 3):
            assert np.array_equal(got, f)
