"""The LU panel kernels of panel.cuh and lu.cuh run on the CPU (fake_cuda/emulate.h: CUDA threads as fibers, the
inline assembly's functions restated): the factors against LAPACK's algorithm in numpy, and what a panel leaves
behind when one of its bounded waits gives up."""
import os
import re
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "hprmat_b200", "csrc")
NB = 32
# inline assembly, restated in emulate.h
RESTATED = ["cp_async_elem", "cp_async_wait_all", "device_ns", "grid_arrive", "grid_wait", "smem_u32", "mbar_init",
            "mbar_try_wait", "mbar_expect_tx", "cluster_arrive", "cluster_wait", "mapa_u32", "st_async16",
            "st_cluster_u32"]


def _without(src, name):
    """src without the definitions of the device function `name`."""
    while True:
        m = re.search(r"^__device__ [^;{}()]*\b" + name + r"\(", src, re.M)
        if not m:
            return src
        i = src.index("{", m.start())
        depth = 0
        for j in range(i, len(src)):
            depth += {"{": 1, "}": -1}.get(src[j], 0)
            if depth == 0:
                break
        src = src[:m.start()] + src[j + 1:]


@pytest.fixture(scope="module")
def emulator(tmp_path_factory):
    d = tmp_path_factory.mktemp("emulator")
    for f in ("common.cuh", "tc_common.cuh", "lu.cuh", "panel.cuh"):
        src = open(os.path.join(CSRC, f)).read()
        for name in RESTATED:
            src = _without(src, name)
        src = re.sub(r'asm volatile\("bar\.sync 1, %0;" ::"r"\((.*?)\) : "memory"\);', r"emu::barrier(1, \1);", src)
        src = re.sub(r'asm volatile\("fence\.mbarrier_init[^;]*;" ::: "memory"\);', "", src)
        src = src.replace("extern __shared__ __align__(16) unsigned char smem_raw[];",
                          "unsigned char* const smem_raw = emu::dynamic_smem;")
        src = src.replace("constexpr unsigned kPanelWaitLimit = 1u << 22;", "#define kPanelWaitLimit emu::wait_limit")
        (d / f).write_text(src)
    (d / "cuda_runtime.h").write_text('#include "emulate.h"\n')
    (d / "cuda.h").write_text("struct CUtensorMap;\ninline uint64_t __cvta_generic_to_shared(const void* p) { return (uint64_t)p; }\n")
    out = str(d / "panels")
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-w", "-pthread", "-I", str(d), "-I",
                    os.path.join(ROOT, "tests", "fake_cuda"), os.path.join(ROOT, "tests", "fake_cuda", "panels.cpp"), "-o", out],
                   check=True)
    return out


class Panel:
    def __init__(self, exe, tmp, kernel, prec, n, k0, ncols, ctas, drop=(-1, -1, 0), limit=1 << 30, flag=0, odd=0):
        f = str(tmp / "out.bin")
        subprocess.run([exe, kernel, prec, *map(str, (n, k0, ncols, ctas, *drop, limit, flag, odd)), f], check=True, timeout=300)
        raw = open(f, "rb").read()
        real, cplx = (np.float64, np.complex128) if prec == "d" else (np.float32, np.complex64)
        ld, sw, self.outside, self.faults = np.frombuffer(raw, np.int32, 4)
        at = [16]

        def take(dtype, count):
            a = np.frombuffer(raw, dtype, count, at[0])
            at[0] += a.nbytes
            return a
        status = take(np.int32, 8)
        self.info, self.timeout = status[0], status[sw]
        self.ipiv = take(np.int32, n)
        lists = take(np.int32, 3 * NB + 1)
        self.top, self.dst, self.src, self.n_extra = lists[:NB], lists[NB:2 * NB], lists[2 * NB:3 * NB], lists[3 * NB]
        self.before = take(cplx, ld * n).reshape(n, ld)[:, :n].T
        self.after = take(cplx, ld * n).reshape(n, ld)[:, :n].T
        self.planes = take(np.float32, 4 * ld * n).reshape(4, n, ld)


def _reference(a, k0, ncols):
    """Unblocked partial pivoting of the panel in double precision: factors, pivots, row order."""
    p = a[k0:, k0:k0 + ncols].astype(np.complex128)
    order, piv = np.arange(k0, len(a)), []
    for j in range(ncols):
        r = j + int(np.argmax(np.abs(p[j:, j].real) + np.abs(p[j:, j].imag)))
        piv.append(k0 + r)
        p[[j, r]], order[[j, r]] = p[[r, j]], order[[r, j]]
        p[j + 1:, j] /= p[j, j]
        p[j + 1:, j + 1:] -= np.outer(p[j + 1:, j], p[j, j + 1:])
    return p, piv, order


@pytest.mark.parametrize("kernel,n,k0,ncols,ctas", [("reg", 40, 8, 32, 1), ("reg", 100, 32, 32, 3), ("reg", 70, 0, 19, 4),
                                                    ("tall", 150, 32, 32, 16), ("grid", 100, 32, 32, 3)])
@pytest.mark.parametrize("prec", ["f", "d"])
def test_factors(emulator, tmp_path, kernel, prec, n, k0, ncols, ctas):
    """Pivots and interchange lists as numpy finds them, factors within 64 m u (u of the type) of the double
    ones; nothing written outside the panel's columns and buffers."""
    q = Panel(emulator, tmp_path, kernel, prec, n, k0, ncols, ctas)
    ref, piv, order = _reference(q.before, k0, ncols)
    assert (q.outside, q.faults, q.timeout, q.info) == (0, 0, 0, 0)
    assert list(q.ipiv[k0:k0 + ncols]) == piv and list(q.top[:ncols]) == list(order[:ncols])
    moved = {int(d): int(s) for d, s in zip(q.dst[:q.n_extra], q.src[:q.n_extra])}
    assert moved == {k0 + i: int(r) for i, r in enumerate(order) if i >= ncols and r != k0 + i}
    u = 2.0 ** -53 if prec == "d" else 2.0 ** -24
    assert np.abs(q.after[k0:, k0:k0 + ncols] - ref).max() <= 64 * (n - k0) * u
    assert np.array_equal(np.delete(q.after, slice(k0, k0 + ncols), 1), np.delete(q.before, slice(k0, k0 + ncols), 1))
    if prec == "f":
        l21 = q.after[k0 + ncols:, k0:k0 + ncols]
        rows = q.planes[:, k0 + ncols:, k0:k0 + ncols]
        assert np.array_equal(rows[0] + rows[1], l21.real) and np.array_equal(rows[2] + rows[3], l21.imag)


# messages lost: all to one CTA; of one CTA to another, from the sixth column on; all to the first CTA from the
# tenth on; none lost, but an earlier panel of the factorisation gave up
LOST = [((-1, 1, 0), 0), ((2, 1, 5), 0), ((-1, 0, 9), 0), ((-1, -1, 0), 9)]


@pytest.mark.parametrize("lost,flag", LOST)
@pytest.mark.parametrize("kernel,n,k0,ncols,ctas", [("reg", 100, 32, 32, 3), ("reg", 130, 0, 32, 4), ("reg", 70, 0, 19, 4),
                                                    ("tall", 150, 32, 32, 16)])
@pytest.mark.parametrize("prec", ["f", "d"])
def test_a_panel_that_gives_up(emulator, tmp_path, kernel, n, k0, ncols, ctas, prec, lost, flag):
    """A lost message makes a bounded wait run out (here after 1000 polls): the panel says so in the status
    word, leaves a list of no interchanges, and writes to no row by a position that it cannot know."""
    q = Panel(emulator, tmp_path, kernel, prec, n, k0, ncols, ctas, lost, 1 << 30 if flag else 1000, flag)
    assert q.timeout == (flag or {"reg": 2, "tall": 3}[kernel])
    assert (q.outside, q.faults) == (0, 0)
    assert q.n_extra == 0 and list(q.top[:ncols]) == list(range(k0, k0 + ncols))
    assert list(q.ipiv[k0:k0 + ncols]) == list(range(k0, k0 + ncols))
    if kernel == "reg":
        assert np.array_equal(q.after, q.before) and not q.planes.any()
    else:  # the sub-panels factor their own rows in place
        assert np.array_equal(np.delete(q.after, slice(k0, k0 + ncols), 1), np.delete(q.before, slice(k0, k0 + ncols), 1))
        assert np.array_equal(q.after[:k0], q.before[:k0])


@pytest.mark.parametrize("prec", ["f", "d"])
def test_a_grid_panel_that_gives_up(emulator, tmp_path, prec):
    """The panel over the whole grid, one CTA missing at its barrier (300 polls): no interchanges, nothing
    written."""
    q = Panel(emulator, tmp_path, "absent", prec, 100, 32, 32, 3, limit=300)
    assert (q.timeout, q.outside, q.faults, q.n_extra) == (1, 0, 0, 0)
    assert list(q.top) == list(q.ipiv[32:64]) == list(range(32, 64))
    assert np.array_equal(q.after, q.before) and not q.planes.any()


@pytest.mark.parametrize("odd", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("kernel,n,k0,ncols,ctas", [("reg", 40, 8, 32, 1), ("reg", 100, 32, 32, 3), ("tall", 150, 32, 32, 16)])
@pytest.mark.parametrize("prec", ["f", "d"])
def test_panels_of_nan_and_infinity(emulator, tmp_path, kernel, n, k0, ncols, ctas, prec, odd):
    """A NaN, an infinity, a column or a whole panel of NaN, a row of infinities: the rows' order stays a
    permutation, no store leaves the buffers, and the panel is not finite where it was not before."""
    q = Panel(emulator, tmp_path, kernel, prec, n, k0, ncols, ctas, odd=odd)
    assert (q.outside, q.faults, q.timeout) == (0, 0, 0)
    order = np.arange(n)
    order[k0:k0 + ncols] = q.top[:ncols]
    order[q.dst[:q.n_extra]] = q.src[:q.n_extra]
    assert sorted(order) == list(range(n))
    assert all(k0 + j <= p < n for j, p in enumerate(q.ipiv[k0:k0 + ncols]))
    assert not np.isfinite(q.after[k0:, k0:k0 + ncols]).all()
    assert np.array_equal(np.delete(q.after, slice(k0, k0 + ncols), 1), np.delete(q.before, slice(k0, k0 + ncols), 1))
