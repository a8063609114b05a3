"""The choices of the decode attention (csrc/attn_route.h), compiled for the host."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "mlx-metal-kernels_b200" / "csrc"


def _run(tmp_path, body):
    (tmp_path / "driver.cpp").write_text('#include "attn_route.h"\n#include <cstdio>\nusing namespace b200q;\nint main() {\n' + body + "\nreturn 0;\n}\n")
    subprocess.run(["g++", "-O1", "-std=c++17", f"-I{CSRC}", str(tmp_path / "driver.cpp"), "-o", str(tmp_path / "driver")], check=True)
    return subprocess.run([str(tmp_path / "driver")], check=True, capture_output=True, text=True).stdout


def test_one_warp_appends_each_row(tmp_path):
    """The cluster kernel's CTAs have eight or sixteen warps: one of them writes the new token's K row, another its V row.  The kernel asks
    nothing but this function."""
    out = _run(tmp_path, "for (int n = 8; n <= 16; n += 8) for (int w = 0; w < n; ++w) std::printf(\"%d %d\\n\", n, (int)append_role(w, n));")
    roles = [tuple(map(int, line.split())) for line in out.splitlines()]
    for warps in (8, 16):
        assert sorted(r for n, r in roles if n == warps) == [0] * (warps - 2) + [1, 2]
    assert "append_role(warp, NW)" in (CSRC / "paged_attn.cu").read_text()
