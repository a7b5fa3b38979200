"""The list of a relayout's pieces when the bins hold more than their peak has (corrupted fills): the
kernels' own rules, compiled for the host, publish no entry that was not written and copy no piece
that leaves the peak's bins."""
import random
import subprocess
from pathlib import Path

import pytest

from pbh_b200.build import nvcc

CSRC = Path(__file__).resolve().parent.parent / "pbh_b200" / "csrc"

# Reads "n nst bins r_off r_size", then per bin "source stay moved destination"; admits each bin as
# layout_peak does and prints entries, published, unwritten among the published, copied outside.
PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "pm_kernels.cuh"
int main() {
  long long n, nst, bins, r_off, r_size;
  while (std::scanf("%lld %lld %lld %lld %lld", &n, &nst, &bins, &r_off, &r_size) == 5) {
    const long long room = piece_room(n, nst);
    std::vector<uint4> list(room);
    std::vector<char> written(room, 0);
    u32 asked = 0;
    for (long long i = 0; i < bins; ++i) {
      u32 src, n0, n1, dst;
      if (std::scanf("%u %u %u %u", &src, &n0, &n1, &dst) != 4) return 1;
      const u32 p = (n0 + MOVE_PIECE - 1) / MOVE_PIECE + (n1 + MOVE_PIECE - 1) / MOVE_PIECE;
      u32 q = asked;
      asked += p;
      if (!piece_fits(q, p, room)) continue;
      const u32 runs[2][2] = {{0, n0}, {n0, n0 + n1}};
      for (auto& r : runs)
        for (u32 k = r[0]; k < r[1]; k += MOVE_PIECE, ++q) {
          list.at(q) = uint4{src + k, dst + k, r[1] - k < MOVE_PIECE ? r[1] - k : MOVE_PIECE, 0};
          written.at(q) = 1;
        }
    }
    const u32 pub = pieces_published(asked, room);
    long long bad = 0, out = 0, moved = 0;
    for (u32 q = 0; q < pub; ++q) {
      if (q >= room || !written[q]) { ++bad; continue; }
      const uint4 m = list[q];
      if (!piece_inside(m.x, m.y, m.z, r_off, r_size)) continue;
      moved += m.z;
      if (m.x < r_off || m.y < r_off || m.x + (long long)m.z > r_off + r_size || m.y + (long long)m.z > r_off + r_size) ++out;
    }
    std::printf("%lld %u %lld %lld %lld\n", room, pub, bad, out, moved);
  }
}
"""


@pytest.fixture(scope="module")
def lists(tmp_path_factory):
    try:
        compiler = nvcc()
    except RuntimeError:
        pytest.skip("nvcc not found")
    d = tmp_path_factory.mktemp("pieces")
    (d / "t.cu").write_text(PROGRAM)
    subprocess.run([compiler, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-I", str(CSRC),
                    "-o", str(d / "t"), str(d / "t.cu")], check=True, capture_output=True, text=True)

    def run(n, nst, r_off, r_size, bins):
        text = f"{n} {nst} {len(bins)} {r_off} {r_size}\n" + "\n".join(" ".join(map(str, b)) for b in bins)
        out = subprocess.run([str(d / "t")], input=text, check=True, capture_output=True, text=True).stdout
        return [int(v) for v in out.split()]
    return run


@pytest.mark.parametrize("n,nst", [(7, 1), (1024, 1), (5000, 8), (100000, 64)])
def test_bins_that_agree_with_their_peak_all_move(lists, n, nst):
    rng = random.Random(n)
    cuts = sorted(rng.randint(0, n) for _ in range(2 * nst - 1))
    runs = [b - a for a, b in zip([0] + cuts, cuts + [n])]
    bins, at = [], 96
    for i in range(nst):
        bins.append((at, runs[2 * i], runs[2 * i + 1], at + n))
        at += runs[2 * i] + runs[2 * i + 1]
    room, published, unwritten, outside, moved = lists(n, nst, 96, 2 * n, bins)
    assert published <= room and (unwritten, outside, moved) == (0, 0, n)


@pytest.mark.parametrize("n,nst", [(7, 1), (5000, 8), (100000, 64)])
def test_bins_that_claim_too_much_copy_nothing_unwritten(lists, n, nst):
    rng = random.Random(n)
    for scale in (2, 20, 1000):
        bins = [(rng.randint(0, 3 * n), rng.randint(0, scale * n), rng.randint(0, n), rng.randint(0, 3 * n))
                for _ in range(nst)]
        bins[rng.randrange(nst)] = (96, scale * n + 1025 * (n // 1024 + 2 * nst), 0, 96)   # more than the list holds
        room, published, unwritten, outside, _ = lists(n, nst, 96, 2 * n, bins)
        assert (published, unwritten, outside) == (0, 0, 0)


def test_a_piece_outside_the_peak_s_bins_is_left_out(lists):
    # two bins, one naming slots of another peak on each side
    room, published, unwritten, outside, moved = lists(4000, 4, 1000, 4000, [
        (900, 50, 0, 2000), (1000, 50, 0, 4990), (4990, 20, 0, 1000), (1000, 60, 0, 4940)])
    assert (published, unwritten, outside, moved) == (4, 0, 0, 60)
