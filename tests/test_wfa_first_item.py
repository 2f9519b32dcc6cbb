"""Which item each block of the WFA block kernel begins with."""
import os
import subprocess

from fake_cuda import HERE, fake_path  # noqa: F401
from genoaligner_gb300 import _build


def test_every_first_item_is_one_blocks(fake_path, tmp_path):
    exe = str(tmp_path / "first_item")
    subprocess.run([_build.nvcc(), *_build.ARCH, *_build.FLAGS, "-cudart", "none", "-o", exe,
                    os.path.join(HERE, "first_item_check.cu"), fake_path], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n", (r.returncode, r.stdout, r.stderr)
