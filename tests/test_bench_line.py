"""bench.py prints its line where the reference's library is not built as well."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_unavailable_names_the_library(monkeypatch):
    import bench
    from oracle import oracle as O
    monkeypatch.setattr(O, "ref_available", lambda native_rng=False: False)
    assert bench.reference_unavailable() == "oracle/_ref/libglimpse_ref.so not built"
    assert bench.reference_unavailable(True) == "oracle/_ref/libglimpse_ref_native.so not built"
    monkeypatch.setattr(O, "ref_available", lambda native_rng=False: True)
    assert bench.reference_unavailable() is None


@pytest.mark.gpu
def test_bench_line_with_and_without_the_reference():
    out = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--config", "small", "--steps", "1",
                          "--warmup", "3"], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
    line = json.loads(out.stdout.strip().splitlines()[-1])
    assert line["unit"] == "samples/s" and line["value"] > 0 and line["e2e"]["value"] > 0 and line["gpu_launches"] > 0
    from oracle import oracle as O
    assert ("value" in line["cpu_baseline"]) == O.ref_available()
