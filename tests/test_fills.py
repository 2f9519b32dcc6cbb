"""A batch's first kernel takes a fixed number of fills; one too many is an error of the
call, not a write past the list."""
import os
import subprocess

from fake_cuda import HERE, fake_path  # noqa: F401
from genoaligner_gb300 import _build


def test_one_fill_too_many_is_refused(fake_path, tmp_path):
    exe = str(tmp_path / "fills")
    subprocess.run([_build.nvcc(), *_build.ARCH, *_build.FLAGS, "-cudart", "none", "-o", exe,
                    os.path.join(HERE, "fills_check.cu"), fake_path], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n", (r.returncode, r.stdout, r.stderr)
