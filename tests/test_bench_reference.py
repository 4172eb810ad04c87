"""The bench's reference arm runs without this library: same weights, made by the oracle."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = """
import sys
import numpy as np
import bench
bench.SHAPES = [("a", 264, 256), ("b", 96, 1024)]
theirs = bench.make_weights(0, by_oracle=True)
assert "librstq" not in open("/proc/self/maps").read(), "the library is loaded"
ours = bench.make_weights(0)
for a, b in zip(theirs, ours):
    for k in ("wq", "ws", "wqi", "wsi", "x"):
        assert np.asarray(a[k]).tobytes() == np.asarray(b[k]).tobytes(), k
"""


def test_the_reference_arm_makes_the_same_weights_without_the_library():
    r = subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
