"""The native operator module (csrc/host/kf_host.cpp): bad arguments end as Python errors, containers may be any object with the attributes, other
threads run while an operator is inside the library."""
import re
from pathlib import Path

import pytest
import torch

gpu = pytest.mark.gpu


def _res_case(M=6, N=128, K=256):
    from lightly_trian_quant_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(1)
    a = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    W = ops.QWeight(torch.randn(N, K, generator=g, device="cuda") * 0.05, "bf16")
    vec = torch.randn(N, generator=g, device="cuda")
    return a, W, vec, torch.randn(M, N, generator=g, device="cuda")


@gpu
@pytest.mark.parametrize("row_map,error", [
    ((0, 5, 2), ZeroDivisionError), ([0, 0, 0], ZeroDivisionError), ((3, 5), ValueError), ((3, 5, 2, 1), ValueError), (7, TypeError),
    ((3.0, 5, 2), TypeError), ((1 << 40, 5, 2), OverflowError), ((4, 5, 1), RuntimeError), ((-3, 5, 2), RuntimeError)])
def test_bad_row_maps_are_python_errors(row_map, error):
    from lightly_trian_quant_b200 import ops

    a, W, vec, res = _res_case()
    with pytest.raises(error):
        ops.gemm_res(a, W, vec, vec, res, out=torch.zeros(2, 5, 128, device="cuda"), row_map=row_map)


@gpu
@pytest.mark.parametrize("kind", [tuple, list, iter])
def test_row_map_takes_any_iterable(kind):
    from lightly_trian_quant_b200 import ops

    a, W, vec, res = _res_case()
    plain = ops.gemm_res(a, W, vec, vec, res)
    out = torch.zeros(2, 5, 128, device="cuda")
    ops.gemm_res(a, W, vec, vec, res, out=out, row_map=kind((3, 5, 2)))
    assert torch.equal(out[:, 2:].reshape(6, 128), plain) and not out[:, :2].any()


@gpu
def test_empty_last_dimension_is_a_python_error():
    from lightly_trian_quant_b200 import ops

    none = torch.zeros(3, 0, device="cuda")
    with pytest.raises(ZeroDivisionError):
        ops.ln_rows(none, none, none, 1e-5)
    with pytest.raises(ZeroDivisionError):
        ops.ln_amax_scale(none, none, none, 1e-5, torch.ones(1, device="cuda"), torch.zeros(2, dtype=torch.int32, device="cuda"))
    with pytest.raises(ZeroDivisionError):
        ops.broadcast_rows(none, torch.zeros(2, 3, 0, device="cuda"), 0)
    with pytest.raises(ops.KfError):
        ops.ln_quant(none, none, none, 1e-5, ops.ActBuf(3, 256, "mx8"))


PROPERTY_PROBE = """
import types
import torch
from lightly_trian_quant_b200 import _lib

log = []

class Rows:
    def __index__(self):
        log.append("used")
        return 128
    def __del__(self):
        log.append("freed")

class Weight:
    K, fmt, sf, ts = 256, "bf16", None, None
    @property
    def N(self):
        return Rows()
    @property
    def q(self):
        return torch.zeros(128, 256, dtype=torch.bfloat16)

try:
    _lib.host().gemm_plain(torch.zeros(1, 256, dtype=torch.bfloat16), Weight(), None, None, 1, 0)
except _lib.KfError as e:
    assert "CUDA" in str(e)
else:
    raise SystemExit("a CPU tensor was taken")
assert log == ["used", "freed"], log
"""


def test_attribute_values_live_until_they_are_used():
    """a container's attribute may be a property whose value nobody else holds (in a process of its own: a use after free may end it)."""
    import subprocess
    import sys
    from pathlib import Path

    from lightly_trian_quant_b200 import build

    build.build()
    r = subprocess.run([sys.executable, "-c", PROPERTY_PROBE], capture_output=True, text=True, cwd=Path(__file__).resolve().parents[1])
    assert r.returncode == 0, (r.returncode, r.stderr)


@gpu
def test_containers_with_property_attributes():
    """operands whose every attribute access makes a new tensor give the bits of the package's own containers."""
    from lightly_trian_quant_b200 import ops

    class Fresh:
        def __init__(self, held):
            self.held = held

        def __getattr__(self, name):
            t = getattr(self.held, name)
            return t.clone() if isinstance(t, torch.Tensor) else t

    g = torch.Generator(device="cuda").manual_seed(2)
    x = torch.randn(300, 512, generator=g, device="cuda").bfloat16()
    a = ops.quant_rows(x, ops.ActBuf(300, 512, "nv4"))
    W = ops.QWeight(torch.randn(384, 512, generator=g, device="cuda") * 0.05, "nv4")
    want = ops.gemm_plain(a, W)
    for _ in range(20):
        assert torch.equal(ops.gemm_plain(Fresh(a), Fresh(W)), want)
    ops.check_device_error()


@gpu
def test_other_threads_run_while_a_launch_waits():
    """a launch blocks while the queue of its stream is full; another Python thread runs meanwhile.  One fp64 product of a few tenths of a second, then
    more launches than the queue holds: the longest gap between the other thread's steps stays far below the longest launch."""
    import threading
    import time

    from lightly_trian_quant_b200 import ops

    n = 16384
    big = torch.ones(n, n, dtype=torch.float64, device="cuda")
    out = torch.empty_like(big)
    x = torch.randn(128, 256, device="cuda")
    buf = ops.ActBuf(128, 256, "mx8")
    ops.quant_rows(x, buf)
    torch.mm(big[:256], big, out=out[:256])                   # the library's first call is out of the way
    torch.cuda.synchronize()
    gaps, stop = [0.0], threading.Event()

    def tick():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            gaps[0] = max(gaps[0], now - last)
            last = now

    t = threading.Thread(target=tick)
    t.start()
    longest = 0.0
    try:
        torch.mm(big, big, out=out)
        for _ in range(3000):
            t0 = time.perf_counter()
            ops.quant_rows(x, buf)
            longest = max(longest, time.perf_counter() - t0)
    finally:
        stop.set()
        t.join()
    torch.cuda.synchronize()
    ops.check_device_error()
    print(f"longest launch {longest * 1e3:.0f} ms, longest gap of the other thread {gaps[0] * 1e3:.1f} ms")
    assert longest > 0.05, "the queue never filled: the test shows nothing"
    assert gaps[0] < 0.5 * longest


def test_no_unordered_state_shared_between_threads():
    """launchers run without the interpreter lock: what they keep between calls is const, per thread, or atomic (PerDevice), never a plain static."""
    csrc = Path(__file__).resolve().parent.parent / "lightly_trian_quant_b200" / "csrc"
    variable = re.compile(r"^\s*static\s+(?!const\b|constexpr\b|thread_local\b|std::atomic\b|PerDevice<|__device__)[\w:<>,* ]+?[\s*&](\w+)\s*(\[[^;]*)?(=[^;]*|\{[^;]*)?;")
    plain = [f"{path.name}:{no}: {line.strip()}" for path in sorted(csrc.rglob("*.c*")) if path.suffix in (".cu", ".cuh", ".cpp")
             for no, line in enumerate(path.read_text().splitlines(), 1) if variable.match(line)]
    assert not plain, plain
