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


USES = {"dense": 0, "append": 1, "window": 2, "plain": 3}


def _choices(tmp_path, queries):
    """(size, preferred) on 148 SMs for queries (B, Hkv, group, walk_pages, use, split, tp_world)."""
    rows = ",".join("{" + ",".join(map(str, (*q[:4], USES[q[4]], int(q[5]), q[6]))) + "}" for q in queries)
    out = _run(tmp_path, "static const int q[][7] = {" + rows + "};\nfor (auto& r : q) {\n"
               "ClusterQuery c = {r[0], r[1], r[2], r[3], (AttnUse)r[4], r[5] != 0, r[6], 0, 0, 148};\n"
               "const ClusterChoice x = cluster_choice(c);\nstd::printf(\"%d %d\\n\", x.size, (int)x.preferred);\n}")
    return [(int(a), b == "1") for a, b in (line.split() for line in out.splitlines())]


def test_long_walks_of_few_heads_go_to_split_kv(tmp_path):
    """Plain pages and windows of few sequences: the cluster kernel up to the walk at which split-KV is measured to be faster.  Dense quantised
    calls, the append, and whoever has no workspace keep the cluster kernel at any length."""
    limits = [(1, 8, 4, 544), (1, 8, 8, 408), (1, 4, 4, 416), (1, 2, 4, 704), (1, 1, 4, 1408), (1, 1, 8, 1056), (1, 3, 4, 288), (2, 4, 4, 572),
              (4, 2, 4, 2024), (3, 4, 4, 832)]
    queries = [(b, kv, g, pages, use, True, 1) for b, kv, g, limit in limits for use in ("plain", "window") for pages in (1, limit, limit + 1, 1 << 27)]
    for i, got in enumerate(_choices(tmp_path, queries)):
        assert got == (8, i % 4 < 2), queries[i]
    unbounded = [(b, kv, g, 1 << 27, use, split, 1) for b, kv, g, _ in limits for use, split in
                 (("dense", True), ("append", True), ("dense", False), ("append", False), ("window", False), ("plain", False))]
    unbounded += [(6, 2, 4, 1 << 27, "plain", True, 1), (13, 1, 8, 1 << 27, "window", True, 1)]
    assert all(got == (8, True) for got in _choices(tmp_path, unbounded))


def test_a_shard_takes_the_kernel_of_the_unsharded_call(tmp_path):
    queries = [(b, kv, g, pages, use, split, 1) for b in (1, 2, 3, 7, 16, 40) for kv in (2, 4, 8, 16) for g in (1, 8) for pages in (1, 40, 128, 256, 420, 560, 2000)
               for use in USES for split in (True, False)]
    shards = [(b, kv // 2, g, pages, use, split, 2) for b, kv, g, pages, use, split, _ in queries]
    assert _choices(tmp_path, queries) == _choices(tmp_path, shards)
