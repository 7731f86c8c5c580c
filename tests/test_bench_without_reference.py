"""The bench where the reference's CPU kernels are neither built nor buildable
(no GPU needed): its reference arm prints one line that says so and ends well,
and the measuring arm has the same reason to put in place of its CPU baseline.
"""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_says_why_it_is_unavailable(tmp_path):
    """In a copy of the tree without oracle/_ref and without the reference's sources."""
    for name in ("bench.py", "paddi_b200", "perf"):
        os.symlink(os.path.join(ROOT, name), tmp_path / name)
    os.mkdir(tmp_path / "oracle")
    for name in ("__init__.py", "oracle.py"):
        (tmp_path / "oracle" / name).write_text(open(os.path.join(ROOT, "oracle", name)).read())
    os.unlink(tmp_path / "bench.py")
    (tmp_path / "bench.py").write_text(open(os.path.join(ROOT, "bench.py")).read())
    env = dict(os.environ, PADDI_REF_SRC=str(tmp_path / "none"))
    out = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--gpus", "1",
                          "--steps", "1", "--warmup", "0"],
                         cwd=tmp_path, env=env, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
    (line,) = [json.loads(v) for v in out.stdout.splitlines()]
    assert line["impl"] == "reference" and "not built" in line["unavailable"]


@pytest.mark.parametrize("built", [True, False])
def test_the_measuring_arm_knows_the_reason(monkeypatch, built):
    sys.path.insert(0, ROOT)
    import bench
    from oracle import oracle as O
    monkeypatch.setattr(O, "ref", lambda: object() if built else None)
    why = bench.reference_missing()
    assert (why is None) if built else ("not built" in why)
