"""The benchmark's reference arm runs without this package's libraries."""
import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_reference_arm_maps_none_of_the_package_libraries():
    code = """
import sys
sys.argv = ["bench.py", "--impl", "reference", "--steps", "1", "--warmup", "1", "--workload", "c3"]
import bench
bench.build_cpu_sample = lambda spec, n: []
bench.cpu_reference_step = lambda *a: (1.0, 1.0)
bench.main()
maps = open("/proc/self/maps").read()
assert "_calls.so" not in maps and "libiflb200" not in maps, "mapped"
assert not any(m.startswith("instinctflash_b200.kernels") for m in sys.modules)
"""
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    assert '"impl": "reference"' in r.stdout
