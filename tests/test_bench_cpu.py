"""bench.py's CPU legs on a machine without the compiled reference: the scalar port is called with whole addresses."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# in a process of its own: an address cut to 32 bits ends it
CHILD = """
import os
import numpy as np
import bench
real = os.path.exists
os.path.exists = lambda p: real(p) and not str(p).endswith("libinferbit_ref.so")
cpu = bench.CpuBaseline()
assert cpu.kind == "port"
rng = np.random.default_rng(1)
keep = np.zeros(1 << 26, np.uint8)                   # large arrays lie above the first 4 GB of addresses
M, N = 64, 1 << 16
w, s, x = rng.integers(-127, 128, (M, N), dtype=np.int8), rng.uniform(0.001, 0.01, M).astype(np.float32), rng.standard_normal(N).astype(np.float32)
out = np.empty(M, np.float32)
cpu.matvec_int8(out, w, s, x, M, N)
assert np.allclose(out, (w.astype(np.float64) @ x) * s, rtol=1e-3, atol=1e-3 * np.abs(x).sum() * s.max())
assert cpu.linear(4, 64, 256, 2, 1e6)["kind"] == "port" and cpu.linear(8, 64, 256, 1, 1e6)["value"] > 0
print("ok")
"""


def test_port_legs_run():
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), (r.returncode, r.stderr[-1000:])


def test_reference_arm_without_the_reference(tmp_path):
    """Without the compiled reference its arm says so; it does not time the port under the reference's name."""
    code = "import os, sys, bench; real = os.path.exists; os.path.exists = lambda p: real(p) and not str(p).endswith('libinferbit_ref.so'); " \
           "sys.argv = ['bench.py', '--impl', 'reference', '--steps', '2', '--warmup', '1']; bench.main()"
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert r.returncode == 0 and line["impl"] == "reference" and "unavailable" in line and "value" not in line
