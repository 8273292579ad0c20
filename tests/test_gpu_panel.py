"""The cluster panel of the LU (panel.cuh): dense solves at the edges of its row split, sub-panels
and cluster sizes, against numpy's solution."""
import ctypes

import numpy as np
import pytest
import torch

from hprmat_b200 import _native as nat
from hprmat_b200 import api

pytestmark = pytest.mark.gpu


def _matrix(n, ties):
    rng = np.random.default_rng(n)
    if ties:  # many equal moduli: the pivot is the lowest such row
        a = rng.integers(-1, 2, (n, n)) + 1j * rng.integers(-1, 2, (n, n)) + 0.01 * rng.uniform(-1, 1, (n, n))
        a[:, : n // 2] = np.round(a[:, : n // 2])
        a += 3.0 * np.sqrt(n) * np.roll(np.eye(n), n // 3, axis=0)
        return a
    return rng.uniform(-1, 1, (n, n)) + 1j * rng.uniform(-1, 1, (n, n))


@pytest.mark.parametrize("ties", [False, True])
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 15, 17, 31, 33, 63, 65, 127, 128, 129, 145, 161, 257, 511, 513, 1025, 2995])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_panel_row_and_column_edges(precision, n, ties):
    """|A X - B| <= 8 n u |A| |X| elementwise maxima (u = 2^-53): the backward error of an LU with
    partial pivoting on these matrices (growth of a few), and of the refined mixed solve."""
    a = _matrix(n, ties)
    b = np.random.default_rng(7 * n).uniform(-1, 1, (n, 3)) + 0j
    with api.Context(precision=precision, max_refine=8, tol=1e-15) as ctx:
        x = ctx.solve_linear(a, b, allow_unconverged=True)
    r = np.abs(a @ x - b).max()
    assert r <= 8 * n * 2.0 ** -53 * np.abs(a).sum(1).max() * np.abs(x).max()


@pytest.mark.parametrize("n,col", [(5, 0), (40, 16), (130, 7), (130, 128), (300, 45), (600, 333)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_zero_column_is_reported(precision, n, col):
    a = _matrix(n, False)
    a[:, col] = 0.0
    with api.Context(precision=precision) as ctx:
        with pytest.raises(api.HprmatError):
            ctx.solve_linear(a, np.ones((n, 1), complex))
        assert ctx.last_stats["info"] == col + 1


@pytest.mark.parametrize("precision,n", [("mixed", 3010), ("mixed", 8192), ("mixed", 8209), ("mixed", 16400),
                                         ("mixed", 24600), ("fp64", 3150), ("fp64", 8209)])
def test_tall_panels(precision, n):
    """Panels of more rows than a cluster's shared memory, at 1 to 4 rows per thread: random
    matrices (pivots all over the rows), the bound of the test above on the GPU."""
    gen = torch.Generator("cuda").manual_seed(n)
    a = torch.complex(*(torch.rand((n, n), dtype=torch.float64, device="cuda", generator=gen) - 0.5 for _ in range(2)))
    b = torch.rand((2, n), dtype=torch.float64, device="cuda", generator=gen).to(torch.complex128)
    x, at = b.clone(), a.T.contiguous()
    torch.cuda.synchronize()
    with api.Context(precision=precision, max_refine=8, tol=1e-15) as ctx:
        ctx.solve_linear_device(at.data_ptr(), x.data_ptr(), n, 2, allow_unconverged=True)
    r = (a @ x.T - b.T).abs().max().item()
    bound = 8 * n * 2.0 ** -53 * a.abs().sum(1).max().item() * x.abs().max().item()
    del a, at
    torch.cuda.empty_cache()  # the largest sizes' memory back for the tests that follow
    assert r <= bound


@pytest.mark.parametrize("n", [257, 385, 1025, 2995, 3333, 6400])
def test_lookahead_leaves_the_factors_alone(n):
    """A trailing matrix updated beside the next panel (from 129 rows on, the default, never): the same
    solution bit for bit, as every element sees the same operations."""
    rng = np.random.default_rng(n)
    a = rng.uniform(-1, 1, (n, n)) + 1j * rng.uniform(-1, 1, (n, n))
    b = rng.uniform(-1, 1, (n, 2)) + 0j
    lib = nat.load()
    xs = []
    with api.Context(precision="mixed", max_refine=8) as ctx:
        for rows in (0, 129, 2048, 129):
            nat.check(lib.hprmat_b200_dev_set_tuning(ctx._h, b"lookahead", rows))
            xs.append(ctx.solve_linear(a, b, allow_unconverged=True))
    for x in xs[1:]:
        assert np.array_equal(x, xs[0])


@pytest.mark.parametrize("precision,nb", [("fp64", 16), ("fp64", 32), ("fp64", 64), ("mixed", 16), ("mixed", 32),
                                          ("mixed", 64), ("mixed", 128)])
def test_block_sizes(precision, nb):
    """U12's substitution at every block size, with ragged last blocks and column tails: the bound of
    the first test."""
    for n in (nb + 1, 2 * nb - 1, 3 * nb + 33, 4 * nb + 64):
        a = _matrix(n, False)
        b = np.random.default_rng(n).uniform(-1, 1, (n, 2)) + 0j
        with api.Context(precision=precision, max_refine=8, tol=1e-15, panel_nb=nb) as ctx:
            x = ctx.solve_linear(a, b, allow_unconverged=True)
        assert np.abs(a @ x - b).max() <= 8 * n * 2.0 ** -53 * np.abs(a).sum(1).max() * np.abs(x).max()


@pytest.mark.parametrize("n", [193, 257, 385, 1025, 3333])
def test_fp64_lookahead(n):
    """The FP64 LU's pairs of block steps (look-ahead from 65 rows on, the default): the first test's bound,
    and the same bits from a second run."""
    a, lib = _matrix(n, False), nat.load()
    b = np.random.default_rng(n).uniform(-1, 1, (n, 2)) + 0j
    xs = {}
    with api.Context(precision="fp64") as ctx:
        for rows in (260, 2048, 260, 2048):
            nat.check(lib.hprmat_b200_dev_set_tuning(ctx._h, b"lookahead", rows))
            x = ctx.solve_linear(a, b)
            assert np.abs(a @ x - b).max() <= 8 * n * 2.0 ** -53 * np.abs(a).sum(1).max() * np.abs(x).max()
            assert np.array_equal(xs.setdefault(rows, x), x)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_block_sizes_in_one_context(precision):
    """One context at several block sizes in turn, on clusters of 16 CTAs each: the bound of the first test."""
    n = 600
    a = _matrix(n, False)
    b = np.random.default_rng(n).uniform(-1, 1, (n, 2)) + 0j
    with api.Context(precision=precision, max_refine=8, tol=1e-15) as ctx:
        for nb in (64, 32, 16, 64) if precision == "fp64" else (128, 64, 32, 16, 128):
            ctx.opts.panel_nb = nb
            nat.check(nat.load().hprmat_b200_set_opts(ctx._h, ctypes.byref(ctx.opts)))
            x = ctx.solve_linear(a, b, allow_unconverged=True)
            assert np.abs(a @ x - b).max() <= 8 * n * 2.0 ** -53 * np.abs(a).sum(1).max() * np.abs(x).max()


@pytest.mark.parametrize("value", [np.nan, np.inf, complex(0.0, -np.inf)])
@pytest.mark.parametrize("n", [100, 400, 1500, 3333])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_nan_and_infinity(precision, n, value):
    """One entry that is not finite, in the first panel, in U12 or in the last rows: the call ends, with an error
    or a solution (for a NaN one that is not finite; an infinite pivot has a finite limit), and the context solves
    the next system to the first test's bound."""
    a = _matrix(n, False)
    b = np.random.default_rng(n).uniform(-1, 1, (n, 1)) + 0j
    with api.Context(precision=precision, max_refine=8, tol=1e-15) as ctx:
        for i, j in ((n // 2, 3), (5, n - 2), (n - 1, n - 1)):
            bad = a.copy()
            bad[i, j] = value
            try:
                x = ctx.solve_linear(bad, b, allow_unconverged=True)
            except api.HprmatError as e:
                assert e.status in (nat.SINGULAR, nat.PIVOT_GROWTH)
            else:
                assert not (np.isnan(value) and np.isfinite(x).all())
        x = ctx.solve_linear(a, b, allow_unconverged=True)
    assert np.abs(a @ x - b).max() <= 8 * n * 2.0 ** -53 * np.abs(a).sum(1).max() * np.abs(x).max()
