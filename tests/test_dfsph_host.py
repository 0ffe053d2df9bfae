"""Host side of the DFSPH pressure solves (no GPU): memory of the cached pair gradients."""
import subprocess
from pathlib import Path

import pytest
import torch

from warpsph_b200 import _capi, build, ops
from warpsph_b200.core import AdjacencyList


class FakeLib:
    """Records the solves that reach the library, with their arguments."""

    def __init__(self):
        self.calls = []

    def sph_dfsph_gradient_bytes(self, n, entries, dim):
        return 16 * (n + entries)

    def __getattr__(self, name):
        return lambda *args: self.calls.append((name, args)) or 0


@pytest.fixture
def host(monkeypatch):
    lib = FakeLib()
    monkeypatch.setattr(_capi, "lib", lambda: lib)
    for name in ("ptr", "fptr", "iptr"):
        monkeypatch.setattr(ops, name, lambda t: None if t is None else t.data_ptr())
    monkeypatch.setattr(ops, "stream_ptr", lambda device: 0)
    monkeypatch.setattr(ops, "_jacobi_workspace", lambda n, d, device: torch.empty(256, dtype=torch.uint8))
    return lib


def solve(adj, n=5):
    cfg = _capi.SphJacobiConfig()
    cfg.max_iterations = 2
    params = _capi.SphParams()
    params.dim = 3
    f, f3 = torch.zeros(n), torch.zeros(n, 3)
    return ops.jacobi_solve(params, ops.DENSITY, cfg, f3, f, f, f, f3, f3, f, 1e-3, adj)


def rows_of(n=5, nnz=20, length=20):
    return AdjacencyList(neighborOffsets=torch.arange(0, 4 * n, 4, dtype=torch.int32), numNeighbors=torch.full((n,), 4, dtype=torch.int32),
                         neighborList=torch.zeros(length, dtype=torch.int32), numRows=n, numCols=n, nnz=nnz)


def test_kept_rows_are_rewritten_before_the_optional_buffer(host, monkeypatch):
    """On a device that is nearly full the rewrite of a kept list must not find its memory taken by the
    gradients, without which the solve still runs."""
    order = []
    adj = rows_of()
    adj._pending = object()

    def rewrite(a, *rest):
        order.append("rows")
        a._pending = None

    monkeypatch.setattr(ops, "_materialize_inter", rewrite)
    monkeypatch.setattr(ops, "_gradient_buffer", lambda *a: order.append("gradients"))
    solve(adj)
    assert order == ["rows", "gradients"]
    assert [name for name, _ in host.calls] == ["sph_dfsph_density_solve"]


def test_the_buffer_covers_the_list_and_not_the_stated_count(host, monkeypatch):
    """The preparation writes one gradient per row entry.  Rows may lie anywhere in the list that they index,
    whatever count a caller's AdjacencyList states."""
    asked = []
    monkeypatch.setattr(ops, "_gradient_buffer", lambda n, entries, d, device: asked.append(entries) or torch.empty(16 * (n + entries), dtype=torch.uint8))
    solve(rows_of(nnz=3, length=32))
    assert asked == [32]
    (name, args), = host.calls
    assert name == "sph_dfsph_solve_cached" and args[4] == 32


def test_a_buffer_that_did_not_fit_is_not_tried_again_until_there_is_room(host, monkeypatch):
    """Each failing allocation flushes the allocator's cache and synchronises, so it happens once."""
    device = torch.device("cuda", 0)
    monkeypatch.setattr(ops, "_gradient_refused", {})
    free, tried = [1000], []

    def empty(size, dtype=None, device=None):
        tried.append(size)
        if size > free[0]:
            raise torch.cuda.OutOfMemoryError("out of memory")
        return ("buffer", size)

    monkeypatch.setattr(ops.torch, "empty", empty)
    monkeypatch.setattr(ops.torch.cuda, "mem_get_info", lambda device: (free[0] - 300, 1 << 30))
    monkeypatch.setattr(ops.torch.cuda, "get_per_process_memory_fraction", lambda device: 1.0)
    monkeypatch.setattr(ops.torch.cuda, "memory_stats", lambda device: {
        "reserved_bytes.all.current": 900, "active_bytes.all.current": 500, "inactive_split_bytes.all.current": 100})
    big, small = 16 * (10 + 90), 16 * (10 + 20)
    assert ops._gradient_buffer(10, 90, 3, device) is None and tried == [big]
    for _ in range(3):
        assert ops._gradient_buffer(10, 90, 3, device) is None
    assert ops._gradient_buffer(10, 200, 3, device) is None
    assert tried == [big]
    # a smaller solve is unaffected, and the large one is served again once memory is back
    assert ops._gradient_buffer(10, 20, 3, device) == ("buffer", small)
    free[0] = 2000
    assert ops._gradient_buffer(10, 90, 3, device) == ("buffer", big)
    assert ops._gradient_refused == {}


def test_blocks_of_a_persistent_launch(tmp_path):
    """A kernel that keeps one particle per group for the whole solve is launched only when all particles fit
    in one round of co-resident blocks, and no launch has more blocks than slots for their partial sums."""
    root = Path(__file__).resolve().parent
    exe = tmp_path / "persistent_grid_check"
    subprocess.run([build.nvcc(), "-std=c++17", "-I", str(build.INCLUDE), "-I", str(build.CSRC), "-o", str(exe),
                    str(root / "native" / "persistent_grid_check.cu")], check=True, capture_output=True)
    cases = [((4736, 32, 296, 2048, 1), 148), ((4736, 32, 148, 2048, 1), 148), ((4736, 32, 147, 2048, 1), 0), ((4737, 32, 148, 2048, 1), 0),
             ((18944, 64, 296, 2048, 1), 296), ((18944, 64, 148, 2048, 1), 0), ((18944, 64, 148, 2048, 0), 148), ((1, 64, 296, 2048, 1), 1),
             ((1 << 29, 64, 592, 2048, 0), 592), ((1 << 29, 64, 4096, 2048, 0), 2048), ((1 << 29, 64, 4096, 1 << 62, 0), 4096),
             ((200000, 64, 4096, 2048, 1), 0)]
    out = subprocess.run([str(exe), *[str(v) for args, _ in cases for v in args]], check=True, capture_output=True, text=True).stdout.split()
    assert [int(v) for v in out] == [want for _, want in cases]
