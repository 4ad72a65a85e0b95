"""The 1080p clip of the benchmark is kept encoded, so that its CPU reference arm needs no encoder."""
import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent

CODE = """
import subprocess, sys
sys.path[:0] = [%r, %r]
def no_child(*a, **k):
    raise SystemExit("a child process was started")
subprocess.run = subprocess.Popen = no_child
from govid_gb300 import workloads
import ebiv_container
clip = workloads.load([workloads.single_1080()])[0]
print(len(clip), len(ebiv_container.packets(clip)), "libebivgpu" in open("/proc/self/maps").read())
"""


def test_the_reference_arm_has_its_clip_without_an_encoder(tmp_path):
    # With an empty content cache: the kept clip is that of the present encoder sources and parameters.
    r = subprocess.run([sys.executable, "-c", CODE % (str(ROOT), str(ROOT / "oracle"))], cwd=str(ROOT), text=True,
                       capture_output=True, timeout=120, env={"EBIV_CONTENT_DIR": str(tmp_path), "PATH": "/usr/bin:/bin"})
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.split() == ["1325127", "300", "False"]
