"""The library's host code on a stand-in CUDA runtime (fake_cuda/runtime.cpp): what is launched, copied and
waited for on which stream, and what an entry point answers when a launch fails or a wait inside a kernel has
given up.  Kernels do not run; a scenario writes the few values that the host code reads from them.  Each scenario
is a process of its own, so that no test meets the real runtime and the stand-in together."""
import ctypes
import os
import shutil
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = os.path.join(ROOT, "tests", "fake_cuda", "runtime.cpp")
WAIT_SITE = 77  # the site a tensor-core wait reports in the error word


class Op(ctypes.Structure):
    _fields_ = [("kind", ctypes.c_char_p), ("name", ctypes.c_char_p), ("stream", ctypes.c_ulonglong),
                ("args", ctypes.POINTER(ctypes.c_void_p)), ("size", ctypes.c_ulonglong), ("grid", ctypes.c_int),
                ("cluster", ctypes.c_int), ("completion_event", ctypes.c_int)]

    def arg(self, i, ctype):
        return ctypes.cast(self.args[i], ctypes.POINTER(ctype))[0]


class Runtime:
    """The stand-in, loaded in front of the library: `ops` lists (kind, name, stream, size, cluster) in
    order; `on_launch(name, op)` may write a kernel's results and return an error code."""

    def __init__(self, lib_path):
        self.ops, self.on_launch, self.error_word = [], None, None
        self._fake = ctypes.CDLL(lib_path, mode=ctypes.RTLD_GLOBAL)
        self._hook = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.POINTER(Op))(self._called)
        self._fake.fake_set_hook(self._hook)
        sys.path.insert(0, ROOT)
        from hprmat_b200 import _native, api, workloads
        self.api, self.nat, self.workloads = api, _native, workloads

    def _called(self, p):
        op = p[0]
        kind, name = op.kind.decode(), op.name.decode()
        self.ops.append((kind, name, op.stream, op.size, op.cluster))
        if kind == "malloc" and op.size == 4:  # the tensor-core kernels' error word is the one such block
            self.error_word = ctypes.cast(op.args[0], ctypes.POINTER(ctypes.c_int))
        if kind == "launch" and self.on_launch:
            return self.on_launch(name, op) or 0
        return 0

    def tune(self, ctx, key, value):
        self.nat.check(self.nat.load().hprmat_b200_dev_set_tuning(ctx._h, key, value))

    def norms(self, values):
        """on_launch part: the column norms' kernel answers with Frobenius norms from `values`, in turn."""
        left = list(values)

        def handle(name, op):
            if "colnorm2_kernel" in name:
                out = ctypes.cast(op.arg(3, ctypes.c_void_p), ctypes.POINTER(ctypes.c_double))
                v = left.pop(0)
                for q in range(op.grid):
                    out[q] = v * v / op.grid
        return handle


def _wait_gives_up_in_the_last_solve(rt):
    """on_launch part: the correction after the residual rule adds a solve whose wait has given up."""
    def handle(name, op):
        if "add_f2d_kernel" in name:
            rt.error_word[0] = WAIT_SITE
    return handle


def last_solve_of_a_dense_call(rt):
    # norms: of B, of the residual of the factors' solution, of the corrected one (below tol, not zero)
    norms, gives_up = rt.norms([1.0, 1e-6, 1e-14]), _wait_gives_up_in_the_last_solve(rt)
    rt.on_launch = lambda name, op: norms(name, op) or gives_up(name, op)
    ctx = rt.api.Context(precision="mixed")
    with pytest.raises(rt.nat.HprmatError) as e:
        ctx.solve_rmatrix(np.eye(200), np.ones(100), 2, 100)
    assert e.value.status == rt.nat.ERR_TIMEOUT and str(WAIT_SITE) in str(e.value)
    rt.on_launch = rt.norms([1.0, 1e-14])
    ctx.solve_rmatrix(np.eye(200), np.ones(100), 2, 100)  # the next call's result is its own


def last_solve_of_an_interval(rt):
    # residual, its rounding scale, residual of the corrected solution; then the second interval
    norms, gives_up = rt.norms([1e-6, 1.0, 1e-14] * 2), _wait_gives_up_in_the_last_solve(rt)
    seen = []

    def on_launch(name, op):
        norms(name, op)
        if "add_f2d_kernel" in name:
            seen.append(name)
            if len(seen) == 2:
                gives_up(name, op)
        if "propagate_kernel" in name:  # garbage in, a zero pivot out
            ctypes.cast(op.arg(9, ctypes.c_void_p), ctypes.POINTER(ctypes.c_int))[0] = 1
    rt.on_launch = on_launch
    ctx = rt.api.Context(precision="mixed")
    w = rt.workloads.small()
    cpot = np.concatenate([w.cpot, w.cpot])
    with pytest.raises(rt.nat.HprmatError) as e:
        ctx.rmatrix(w.nch, w.lval, w.qk, w.eta, w.rmax, w.nr, 2, cpot)
    assert len(seen) == 2
    assert e.value.status == rt.nat.ERR_TIMEOUT and str(WAIT_SITE) in str(e.value)


def error_beside_a_panel(rt):
    """The look-ahead's panel is on its own stream when a launch beside it fails: the call does not return
    while that panel may still write into the matrix."""
    for prec, n in (("mixed", 700), ("fp64", 700)):
        state = {}

        def on_launch(name, op):
            if state.get("panel") and op.stream != state["panel"]:
                state["failed"] = True
                return 1
            if op.completion_event:  # the panel beside which the update runs
                state["panel"] = op.stream
        ctx = rt.api.Context(precision=prec)
        rt.tune(ctx, b"lookahead", 512)
        rt.on_launch = on_launch
        with pytest.raises(rt.nat.HprmatError) as e:
            ctx.solve_linear(np.eye(n), np.ones((n, 1)))
        assert state.get("failed") and e.value.status == rt.nat.ERR_CUDA
        mine = [o for o in rt.ops if o[2] == state["panel"]]
        assert mine[-1][0] == "sync", mine[-1]


def a_launch_error_is_reported_once(rt):
    """The runtime also keeps a failed launch's error for cudaGetLastError; the next call on the thread must not
    find it there."""
    def solve(prec):
        ctx = rt.api.Context(precision=prec)
        rt.on_launch = rt.norms([1.0, 1e-14])
        ctx.solve_linear(np.eye(300), np.ones((300, 1)))
    for prec, kernel in (("mixed", "panel_reg_kernel"), ("fp64", "zgemm_dmma_kernel"), ("mixed", "full_inverse_kernel")):
        failed = []
        rt.on_launch = lambda name, op: failed.append(name) or 1 if kernel in name and not failed else 0
        ctx = rt.api.Context(precision=prec)
        with pytest.raises(rt.nat.HprmatError) as e:
            ctx.solve_linear(np.eye(300), np.ones((300, 1)))
        assert failed and e.value.status == rt.nat.ERR_CUDA
        solve("mixed")
        solve("fp64")


def block_sizes_in_turn(rt):
    """One context that factorises at one block size and then at another: each is a panel kernel of its own,
    and launches on clusters of more than 8 CTAs."""
    for prec in ("mixed", "fp64"):
        sizes = (128, 64, 32, 16) if prec == "mixed" else (64, 32, 16)
        ctx = rt.api.Context(precision=prec)
        for nb in sizes + sizes[::-1]:
            ctx.opts.panel_nb = nb
            rt.nat.check(rt.nat.load().hprmat_b200_set_opts(ctx._h, ctypes.byref(ctx.opts)))
            rt.on_launch = rt.norms([1.0, 1e-14])
            del rt.ops[:]
            ctx.solve_linear(np.eye(600), np.ones((600, 1)))
            assert max(o[4] for o in rt.ops if "panel_reg_kernel" in o[1]) == 16


def scan_workers_take_the_look_ahead(rt):
    """`lookahead` 0 on a context holds for the workers of its scans: no panel beside an update, no stream for
    it."""
    for rows in (512 * 4, 0):
        w = rt.workloads.production(nch=12, nr=60, rmax=20.0, energy=5.0)
        ctx = rt.api.Context(precision="fp64")
        rt.tune(ctx, b"lookahead", rows)
        beside = []
        rt.on_launch = lambda name, op: beside.append(name) if op.completion_event else 0
        ctx.rmatrix_scan([(w.lval, w.cpot, np.array([w.qk] * 2), np.array([w.eta] * 2))], 20.0, 60, nworkers=2)
        assert bool(beside) == (rows > 0)


def workers_of_the_shifted_scan(rt):
    """`hess_workers` bounds the blocks in flight: three blocks of one order take three workers of 3, one of
    1; blocks of 4, 13 and 24 channels, the largest of which is most of the work, take two."""
    def workers(channels, limit):
        blocks = []
        for nch in channels:
            w = rt.workloads.production(nch=nch, nr=60, rmax=20.0, energy=5.0)
            blocks.append((w.lval, w.cpot, np.array([w.qk]), np.array([w.eta])))
        ctx = rt.api.Context(precision="mixed")
        rt.tune(ctx, b"hess_workers", limit)
        del rt.ops[:]
        ctx.rmatrix_scan(blocks, 20.0, 60, method="shifted", raise_on_unit_error=False)
        return len({o[2] for o in rt.ops if "hb_gemv_kernel" in o[1]})
    assert [workers((9, 9, 9), n) for n in (1, 2, 3)] == [1, 2, 3]
    assert workers((4, 13, 24), 3) == 2


SCENARIOS = {f.__name__: f for f in (last_solve_of_a_dense_call, last_solve_of_an_interval, error_beside_a_panel,
                                   a_launch_error_is_reported_once, block_sizes_in_turn,
                                   scan_workers_take_the_look_ahead, workers_of_the_shifted_scan)}


@pytest.fixture(scope="module")
def stand_in(tmp_path_factory):
    from hprmat_b200 import build
    include = os.path.join(os.path.dirname(shutil.which(build.nvcc())), "..", "include")
    out = str(tmp_path_factory.mktemp("fake_cuda") / "libfake_cuda.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", include, SOURCE, "-o", out], check=True)
    return out


@pytest.mark.parametrize("scenario", sorted(SCENARIOS))
def test_host_path(stand_in, scenario):
    r = subprocess.run([sys.executable, os.path.abspath(__file__), stand_in, scenario], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


if __name__ == "__main__":
    SCENARIOS[sys.argv[2]](Runtime(sys.argv[1]))
