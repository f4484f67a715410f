"""The reduction's map from a thread to its two elements of an 8 x 8 x 8 block
(orbit_coords, compiled for the host from the kernels' own header), enumerated:
every element is met once, no shared-memory read of a half-warp hits a bank pair
twice, and the lanes that the fixed shuffles add up are those of equal coordinates."""
import itertools
import subprocess

import pytest

from libcc_b200 import build as B

MAIN = """
#include "cct_reduce_block.cuh"
int main() {
  for (int t = 0; t < cct::red::RT; t++) std::printf("%d\\n", cct::red::orbit_coords(t));
}
"""


@pytest.fixture(scope="module")
def coords(tmp_path_factory):
    """coords[thread] = (l0, l1, l2) of its first element; the second has l2 ^ 4."""
    d = tmp_path_factory.mktemp("orbit")
    (d / "main.cu").write_text(MAIN)
    subprocess.run([B.nvcc(), *B.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I", str(B.CSRC), "-I",
                    str(B.ROOT / "include"), str(d / "main.cu"), "-o", str(d / "main")], check=True,
                   capture_output=True)
    out = subprocess.run([str(d / "main")], check=True, capture_output=True, text=True).stdout.split()
    packed = [int(v) for v in out]
    assert len(packed) == 256 and all(0 <= v < 512 for v in packed)
    return [(v & 7, v >> 3 & 7, v >> 6) for v in packed]


def test_every_element_of_a_block_once(coords):
    seen = {(a, b, c ^ 4 * e) for a, b, c in coords for e in (0, 1)}
    assert seen == set(itertools.product(range(8), repeat=3))


def test_half_warp_reads_hit_sixteen_bank_pairs(coords):
    for first in range(0, 256, 16):
        for e in (0, 1):
            lanes = [(a, b, c ^ 4 * e) for a, b, c in coords[first:first + 16]]
            for p in itertools.permutations(range(3)):  # X: element (u0, u1, u2) at 64 u0 + 8 u1 + u2
                assert len({(64 * x[p[0]] + 8 * x[p[1]] + x[p[2]]) % 16 for x in lanes}) == 16
            for u, v in itertools.permutations(range(3), 2):  # VOE tiles: entry (u, v) at u + 8 v
                assert len({(x[u] + 8 * x[v]) % 16 for x in lanes}) == 16


@pytest.mark.parametrize("axis,masks,writers", [(0, (1, 16), 17), (1, (2, 24), 18), (2, (4, 16), 20)])
def test_shuffles_add_the_lanes_of_equal_coordinates(coords, axis, masks, writers):
    """After the two xor shuffles a lane holds the sum over its four lanes of equal
    coordinate, and the lanes that write (no bit of `writers`) are one per value."""
    for warp in range(8):
        l = [coords[32 * warp + lane][axis] for lane in range(32)]
        for lane in range(32):
            group = {lane, lane ^ masks[0], lane ^ masks[1], lane ^ masks[0] ^ masks[1]}
            assert len(group) == 4 and {q for q in range(32) if l[q] == l[lane]} == group
        assert sorted(l[lane] for lane in range(32) if lane & writers == 0) == list(range(8))


def test_second_element_of_lane_xor_8_has_the_same_l2(coords):
    for t, (_, _, c) in enumerate(coords):
        assert coords[t ^ 8][2] ^ 4 == c
