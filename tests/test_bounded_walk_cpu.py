"""Control flow around waits that may give up (csrc/bounded_walk.hpp), compiled for the host: threads stand for warps."""
import re
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

PROGRAM = r"""
#include "bounded_walk.hpp"
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <thread>
#include <vector>

// a barrier of N threads that reports who waits in vain, with the conjunction of what they bring
struct Barrier {
    static constexpr int N = 4;
    std::mutex m;
    std::condition_variable cv;
    int here = 0, round = 0;
    bool all = true, result = true;
    bool meet(bool v) {
        std::unique_lock<std::mutex> l(m);
        const int r = round;
        all = all && v;
        if (++here == N) {
            result = all, all = true, here = 0, round++;
            cv.notify_all();
        } else if (!cv.wait_for(l, std::chrono::seconds(5), [&] { return round != r; })) {
            printf("a warp waits for others that have left\n");
            exit(1);
        }
        return result;
    }
};

int main() {
    // warp `w` gives up at its `at`-th tile of seven
    for (int w = 0; w < Barrier::N; w++)
        for (int at = 0; at <= 7; at++) {
            Barrier b;
            bool ok[Barrier::N];
            int done[Barrier::N] = {};
            std::vector<std::thread> t;
            for (int i = 0; i < Barrier::N; i++)
                t.emplace_back([&, i] {
                    ok[i] = rnb::walk_tiles(2, 3, 23, [&](int n) { return !(i == w && n == at); }, [&](bool v) { return b.meet(v); },
                                            [&](int tile) {
                                                if (tile != 2 + 3 * done[i]) exit(2);
                                                for (int k = 0; k < 3; k++) b.meet(true);   // the barriers of a tile
                                                done[i]++;
                                            });
                });
            for (auto &x : t) x.join();
            for (int i = 0; i < Barrier::N; i++)
                if (ok[i] != (at == 7) || done[i] != at) return 3;
        }
    return 0;
}
"""


def run(tmp_path, program):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(program)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", str(ROOT / "runnburn_b200" / "csrc"), "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, (r.returncode, r.stdout)


DRAIN = r"""
#include "bounded_walk.hpp"
#include <vector>

int main() {
    for (unsigned ring = 1; ring <= 5; ring++)
        for (unsigned issued = 0; issued <= 4 * ring + 1; issued++) {
            std::vector<int> last(ring, -1), seen(ring, -1);
            for (unsigned i = 0; i < issued; i++) last[i % ring] = (i / ring) & 1;
            rnb::drain_ring(issued, ring, [&](unsigned slot, unsigned parity) { seen.at(slot) = (int)parity; });
            if (seen != last) return 1;
        }
    return 0;
}
"""


def test_drain_waits_for_the_last_fill_of_every_slot(tmp_path):
    run(tmp_path, DRAIN)


@pytest.mark.parametrize("file,kernel", [
    ("dense.cuh", "dense_gemm_pair_kernel"), ("dense.cuh", "dense_gemm_split_kernel"), ("prefill_gemm_split.cuh", "prefill_gemm_split_kernel"),
    ("prefill_gemm_pair.cuh", "prefill_gemm_pair_kernel"), ("prefill_attention_tiled.cuh", "prefill_attention_tiled_kernel"),
    ("causal_attention_tc.cuh", "causal_attention_tc_kernel"),
])
def test_producers_drain_whatever_their_own_waits_returned(file, kernel):
    """Every ring that a kernel announces copies on is drained, and not behind the producer's own outcome (`ok`)."""
    text = (ROOT / "runnburn_b200" / "csrc" / file).read_text()
    body = text[text.index(kernel + "("):]
    body = body[:body.index("\n}\n")]
    drains = re.findall(r"\n(.*)pg_drain\(&?(\w+),", body)
    rings = {"raw_full", "full"} if kernel == "prefill_gemm_pair_kernel" else {"q_full", "kfull", "vfull"} if "causal" in kernel else {"full"}
    assert {d[1] for d in drains} == rings
    assert not any("ok" in d[0] for d in drains)


def test_warps_that_share_barriers_leave_the_tiles_together(tmp_path):
    run(tmp_path, PROGRAM)


@pytest.mark.parametrize("kernel", ["dense_gemm_pair_kernel"])
def test_barriers_between_warps_stand_behind_an_agreed_wait(kernel):
    text = (ROOT / "runnburn_b200" / "csrc" / "dense.cuh").read_text()
    body = text[text.index(kernel + "("):]
    body = body[:body.index("\n}\n")]
    assert body.index("walk_tiles(") < body.index("bar.sync")
