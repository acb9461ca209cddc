"""Batches whose rows an int does not count go to the GPU in several launches:
every image once, and no launch with more rows than an int holds."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "voreen_gb300", "csrc")


def test_images_per_launch(tmp_path):
    cc = shutil.which("g++")
    if cc is None:
        pytest.skip("needs g++")
    cases = [(1, 1), (8, 48), (1, 2 ** 31 - 1), (5, 2 ** 29), (2 ** 31 - 1, 1), (2 ** 31 - 1, 2), (2 ** 20 + 1, 2 ** 11),
             (7, 2 ** 30), (4, 0), (0, 5)]
    src = tmp_path / "rows.cpp"
    src.write_text('#include <cstdio>\n#include "nn_rows.h"\nint main() {\n' +
                   "".join(f'    std::printf("%d\\n", images_per_launch({n}, {r}ll));\n' for n, r in cases) + "}\n")
    subprocess.run([cc, "-I", CSRC, str(src), "-o", str(tmp_path / "rows")], check=True, capture_output=True, text=True)
    got = [int(x) for x in subprocess.run([str(tmp_path / "rows")], capture_output=True, text=True, check=True).stdout.split()]
    for (images, rows), per in zip(cases, got):
        assert 1 <= per <= max(images, 1)
        assert per * rows <= 2 ** 31 - 1
        # as many as there are, or as an int counts
        assert per == max(images, 1) or (per + 1) * rows > 2 ** 31 - 1
