"""The shares of a batch's workers in the GPU (csrc/coop_share.h): every
cooperative launch finds places for all its blocks, wherever the blocks of the
other workers' launches lie."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "realtime_robot_gb300" / "csrc"
MAX_WORKERS = 16


@pytest.fixture(scope="module")
def shares(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("share")
    (d / "s.cpp").write_text('#include "coop_share.h"\n#include <cstdio>\n#include <initializer_list>\nint main() {\n'
                             "  for (int sms : {4, 7, 148, 152}) for (int w = 2; w <= 16; ++w) for (int g = 1; g <= 2; ++g) {\n"
                             "    const auto s = rtr::coop_share(sms, w, g);\n"
                             '    std::printf("%d %d %d %d %d\\n", sms, w, g, s.icp, s.gc);\n  }\n}\n')
    subprocess.run([cxx, "-std=c++17", "-I", str(CSRC), str(d / "s.cpp"), "-o", str(d / "s")], check=True)
    out = subprocess.run([str(d / "s")], capture_output=True, text=True, check=True).stdout
    return {(s, w, g): (i, c) for s, w, g, i, c in (map(int, line.split()) for line in out.splitlines())}


def places_lost(blocks, sms):
    """Most half-SM places that `blocks` quarter-SM blocks can take: one on each
    SM costs a place, and so does every second one after that."""
    return blocks if blocks <= sms else sms + (blocks - sms + 1) // 2


def test_places_lost_by_enumeration():
    def worst(blocks, sms):  # over every distribution of blocks to SMs
        if sms == 0:
            return 0 if blocks == 0 else -10**9
        return max((j + 1) // 2 + worst(blocks - j, sms - 1) for j in range(min(4, blocks) + 1))
    for sms in range(1, 5):
        for blocks in range(4 * sms + 1):
            assert places_lost(blocks, sms) >= worst(blocks, sms)


def test_every_launch_finds_its_places(shares):
    for (sms, workers, gc_per_sm), (icp, gc) in shares.items():
        for k in range(workers + 1):  # workers in the ICP, the others in the grouping
            if gc_per_sm == 2:
                if k < workers:
                    assert (workers - k) * gc <= 2 * sms - places_lost(k * icp, sms), (sms, workers, k)
                assert k * icp <= 4 * sms - 2 * (workers - k) * gc, (sms, workers, k)
            else:  # a block of either kind may spoil its SM
                assert k * icp + (workers - k) * gc <= sms, (sms, workers, k)


def test_shares_use_the_gpu(shares):
    assert shares[152, 4, 2] == (114, 57) and shares[152, 2, 2] == (228, 114) and shares[152, 4, 1] == (38, 38)
    assert all(i >= 1 and g >= 1 for (s, w, _), (i, g) in shares.items() if s >= 148)
