"""Host-side utilities: the clock sampler against a stand-in `nvidia-smi`, the phase timers without a GPU."""
import os
import stat
import time

import pytest
import torch

from dion_b200.utils.clocks import ClockSampler
from dion_b200.utils.timers import PhaseTimers

_FAKE = """#!/bin/sh
# prints what `nvidia-smi --query-gpu=... --format=csv,noheader,nounits -lms N` prints, forever
i=0
while true; do
  if [ $i -lt 2 ]; then echo "0, 345, 1965, 180.5, Not Active, Not Active, Not Active, Not Active";
  else echo "0, 1650, 1965, 951.2, Not Active, Not Active, Not Active, Active"; fi
  i=$((i+1))
  sleep 0.02
done
"""


def test_clock_sampler_reports_clocks_under_load_and_reasons(tmp_path, monkeypatch):
    exe = tmp_path / "nvidia-smi"
    exe.write_text(_FAKE)
    exe.chmod(exe.stat().st_mode | stat.S_IEXEC)
    monkeypatch.setenv("PATH", f"{tmp_path}{os.pathsep}{os.environ['PATH']}")
    s = ClockSampler(gpu_index=0, period_ms=20)
    s.start()
    time.sleep(0.5)
    out = s.stop()
    assert out["samples"] >= 5
    assert out["sm_mhz"] == 1650.0            # the idle samples (low power) do not count
    assert out["sm_max_mhz"] == 1965.0
    assert out["reasons"] == ["sw_power_cap"]
    assert out["power_w_max"] == 951.2


def test_clock_sampler_without_the_tool(monkeypatch, tmp_path):
    monkeypatch.setenv("PATH", str(tmp_path))
    s = ClockSampler()
    s.start()
    assert s.stop() == {"sm_mhz": None, "sm_max_mhz": None, "reasons": [], "samples": 0}


@pytest.mark.skipif(torch.cuda.is_available(), reason="describes the machine without a GPU")
def test_phase_timers_are_inert_without_a_gpu():
    t = PhaseTimers(enabled=True)
    t.start("a")
    t.stop("a")
    assert t.summary() == {} and t.max_over_ranks() == {}


@pytest.mark.parametrize("M,N,K,rows,world", [(512, 96, 64, 256, 2), (2048, 1536, 768, 1024, 2), (8192, 2304, 768, 4096, 2),
                                              (4096, 4096, 1024, 2048, 2), (32768, 1536, 768, 16384, 2),
                                              (65536, 384, 768, 8192, 8), (32768, 768, 768, 4096, 8)])
def test_gather_gemm_plan_invariants(M, N, K, rows, world):
    """Host-side plan of the GEMM that all-gathers its first operand: every tile's rows sit inside one
    readiness chunk of one source rank, tiles are visited own rows first and then in ring order (the order
    in which the copier warps fetch), the copy units tile every chunk exactly, and the counter buffer the
    Python side allocates is large enough."""
    from dion_b200.ops import _ext

    if not _ext.load(required=False):
        pytest.skip("extension not built")
    unit = 64 * 1024
    for rank in range(world):
        plan = list(torch.ops.dion_b200.gemm_gather_plan(M, N, K, rows, world, rank))
        assert plan, "shapes were rejected"
        tile_m, bn, pair, chunk_rows, units_per_chunk, m_rot, tiles_m, tiles_n = plan
        assert tile_m == (256 if pair else 128) and bn in (128, 256)
        assert rows % chunk_rows == 0 and chunk_rows % tile_m == 0 and tiles_m * tile_m == M
        assert 2 + M // chunk_rows <= 2 + M // 128
        ring_seen = []
        for t in range(tiles_m * tiles_n):
            m_blk = (t // tiles_n + m_rot) % tiles_m
            row0 = m_blk * tile_m
            assert row0 % chunk_rows + tile_m <= chunk_rows          # one chunk per tile (both CTAs of a pair)
            src = row0 // rows
            assert (row0 + tile_m - 1) // rows == src                # one source rank per tile
            ring = (src - rank) % world
            if not ring_seen or ring_seen[-1] != ring:
                ring_seen.append(ring)
        assert ring_seen == list(range(world))                       # own rows first, then ring order, each once
        chunk_bytes = chunk_rows * K * 2
        assert units_per_chunk == -(-chunk_bytes // unit)
        covered = 0
        for u in range(units_per_chunk):
            lo, hi = u * unit, min((u + 1) * unit, chunk_bytes)
            assert lo < hi and lo % 16 == 0 and (hi - lo) % 16 == 0
            covered += hi - lo
        assert covered == chunk_bytes


def test_gather_gemm_plan_rejects_ragged_row_blocks():
    from dion_b200.ops import _ext

    if not _ext.load(required=False):
        pytest.skip("extension not built")
    assert list(torch.ops.dion_b200.gemm_gather_plan(400, 96, 64, 200, 2, 0)) == []      # rows not a multiple of 128
    assert list(torch.ops.dion_b200.gemm_gather_plan(512, 96, 64, 256, 3, 0)) == []      # world * rows != M


def _load_benchmark_module(name):
    import importlib.util

    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    spec = importlib.util.spec_from_file_location(name, os.path.join(root, "benchmark", name + ".py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def test_newton_schulz_benchmark_flop_count_and_plot(tmp_path):
    """FLOP accounting of the Newton-Schulz benchmark (4 m^2 n + 2 m^3 per step, the smaller dimension as m,
    as in the reference's script) and its SVG plot writer, which needs no plotting library."""
    bench = _load_benchmark_module("benchmark_newton_schulz")
    assert bench.ns_flops(4, 8, iters=1) == 4 * 16 * 8 + 2 * 64
    assert bench.ns_flops(8, 4, iters=1) == bench.ns_flops(4, 8, iters=1)
    assert bench.ns_flops(4, 8, batch=3, iters=5) == 15 * bench.ns_flops(4, 8, iters=1)
    rows = [{"m": 512, "tcgen05_tflops": 100.0, "torch_tflops": 80.0},
            {"m": 1024, "tcgen05_tflops": 400.0, "torch_tflops": 300.0, "triton_ref_tflops": 350.0}]
    path = tmp_path / "sub" / "ns.svg"
    bench.write_plot(rows, str(path))
    svg = path.read_text()
    assert svg.startswith("<svg") and svg.rstrip().endswith("</svg>")
    assert svg.count("<polyline") == 3 and "reference Triton" in svg and ">1024<" in svg


def test_loss_curve_markov_batches_are_reproducible_and_follow_the_chain():
    lc = _load_benchmark_module("loss_curve")
    a = lc.markov_batches(2, 3, 16, states=8, fanout=2, vocab=50, seed=5)
    b = lc.markov_batches(2, 3, 16, states=8, fanout=2, vocab=50, seed=5)
    assert all(torch.equal(x1, x2) and torch.equal(y1, y2) for (x1, y1), (x2, y2) in zip(a, b))
    x, y = a[0]
    assert x.shape == (3, 16) and torch.equal(x[:, 1:], y[:, :-1])     # targets are the inputs shifted by one
    assert len(torch.unique(torch.cat([x.flatten(), y.flatten()]))) <= 8
    # every token has at most `fanout` distinct successors over all batches
    succ = {}
    for x, y in a:
        for s, t in zip(x.flatten().tolist(), y.flatten().tolist()):
            succ.setdefault(s, set()).add(t)
    assert max(len(v) for v in succ.values()) <= 2


def test_openmp_compiler_selection(tmp_path, monkeypatch):
    """`ensure_openmp_cxx` keeps a compiler that can build OpenMP code and replaces one that cannot."""
    from dion_b200.utils import compilers

    assert compilers.can_openmp("/nonexistent/compiler") is False
    broken = tmp_path / "g++"
    broken.write_text("#!/bin/sh\nexit 1\n")
    broken.chmod(broken.stat().st_mode | stat.S_IEXEC)
    assert compilers.can_openmp(str(broken)) is False
    monkeypatch.setenv("CXX", str(broken))
    chosen = compilers.ensure_openmp_cxx()
    if chosen:                                   # a working compiler exists on this machine
        assert chosen != str(broken) and os.environ["CXX"] == chosen and compilers.can_openmp(chosen)
        monkeypatch.setenv("CXX", chosen)
        assert compilers.ensure_openmp_cxx() == chosen


def test_a_refused_call_raises_a_message_with_numbers_in_it():
    """In a process of its own: with a second C++ library in the extension, printing the strides ends it with a signal."""
    import subprocess
    import sys

    from dion_b200.ops import _ext

    if not _ext.load(required=False):
        pytest.skip("extension not built")
    code = """
import torch
from dion_b200.ops import _ext
_ext.load(required=False)
x = torch.zeros(8, 8)
try:
    torch.ops.dion_b200.gemm_plan(torch.zeros(16, 16)[::2, ::2], x, None, x)
except RuntimeError as e:
    assert "strides = [32, 2]" in str(e), e
    print("raised")
"""
    done = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                          cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert done.returncode == 0 and done.stdout.strip() == "raised", (done.returncode, done.stderr[-500:])


def _kernels():
    """(file, name, body) of every kernel in the sources."""
    import re

    from dion_b200.ops import _ext

    for path in _ext.sources():
        text = path.read_text()
        for m in re.finditer(r"__global__ void(?:\s+__launch_bounds__\((?:[^()]|\([^()]*\))*\))?\s+(\w+)\s*\(", text):
            start = text.index("{", m.end())
            depth, end = 1, start + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            yield path.name, m.group(1), text[start:end]


def test_kernels_that_start_early_wait_before_they_take_tensor_memory():
    """A CTA that holds tensor memory while it waits for the kernel before it could keep that kernel from its own."""
    seen = set()
    for file, name, body in _kernels():
        if "pdl_trigger();" not in body:
            continue
        seen.add(name)
        assert body.count("pdl_wait();") == 1, (file, name)
        if "tmem_alloc" in body:
            assert body.index("pdl_wait();") < body.index("tmem_alloc"), (file, name)
    assert {"gemm_kernel", "attn_fwd_kernel", "attn_bwd_dq_kernel", "attn_bwd_dkv_kernel", "newton_schulz_kernel",
            "cross_entropy_kernel", "adamw_kernel"} <= seen


def test_what_a_kernel_needs_once_per_device(tmp_path):
    """The helper behind every opt-in to large shared memory, against a runtime that only names the current device."""
    import re
    import shutil
    import subprocess

    from dion_b200.ops import _ext

    src = _ext.sources()[0].parent
    for path in src.glob("*.cu"):  # the opt-in belongs to a device: one flag for all of them skips it on the second
        assert not re.search(r"static bool \w+ = false;", path.read_text()), path.name
    cxx, cuda = os.environ.get("CXX", "g++"), os.environ.get("CUDA_HOME", "/usr/local/cuda")
    if not (shutil.which(cxx) and os.path.exists(os.path.join(cuda, "include", "cuda_runtime.h"))):
        pytest.skip("no compiler")
    (tmp_path / "t.cpp").write_text(r"""
#include "per_device.h"
#include <stdio.h>
#include <thread>
static thread_local int current = 0;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = current; return current < 0 ? cudaErrorNoDevice : cudaSuccess; }
int main() {
  std::atomic<unsigned long long> done{0};
  std::atomic<int> calls[80] = {};
  bool fail = true;
  auto on = [&](int dev) {
    current = dev;
    return dion::once_per_device(done, [&] { ++calls[current]; return fail ? cudaErrorInvalidValue : cudaSuccess; });
  };
  bool ok = on(3) == cudaErrorInvalidValue && on(3) == cudaErrorInvalidValue;  // a failure is not remembered
  fail = false;
  for (int round = 0; round < 2; ++round)
    for (int dev : {0, 1, 3, 63, 64, 70}) ok = ok && on(dev) == cudaSuccess;
  ok = ok && calls[0] == 1 && calls[1] == 1 && calls[3] == 3 && calls[63] == 1 && calls[64] == 2 && calls[70] == 2;
  ok = ok && on(-1) == cudaErrorNoDevice;
  std::thread ts[8];
  std::atomic<bool> all{true};
  for (auto& t : ts) t = std::thread([&] { if (on(5) != cudaSuccess || calls[5] == 0) all = false; });
  for (auto& t : ts) t.join();
  puts(ok && all && calls[5] >= 1 ? "ok" : "wrong");
}
""")
    exe = tmp_path / "t"
    subprocess.run([cxx, "-std=c++17", "-pthread", f"-I{src}", f"-I{cuda}/include", str(tmp_path / "t.cpp"), "-o", str(exe)],
                   check=True, capture_output=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True).stdout.strip() == "ok"
