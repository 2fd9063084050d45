"""The placing of chunks in the ring kernels' rings (ring::Placer of
kami_b200/csrc/ring_place.cuh, compiled here) against its definition, for the
FP64 kernel's 32 records and the 16-bit kernel's 16: where each chunk goes, which
one must be done with before, which must have landed."""
import os
import random
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kami_b200", "csrc")
MAIN = """
#include "ring_place.cuh"
#include <cstdio>
int main()
{
    int ring, recs, most, n, bytes;
    while (std::scanf("%d %d %d %d", &ring, &recs, &most, &n) == 4)
    {
        kami::ring::Placer p(ring, recs, most);
        p.place(ring, &bytes, &bytes); // what an earlier list leaves is cleared
        p.clear();
        for (int dep, land; n--;)
        {
            if (std::scanf("%d", &bytes) != 1)
                return 1;
            const int at = p.place(bytes, &dep, &land);
            std::printf("%d %d %d\\n", at, dep, land);
        }
    }
}
"""


@pytest.fixture(scope="module")
def placer(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("place")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=undefined", "-fno-sanitize-recover=all", "-I", CSRC,
                    str(d / "main.cpp"), "-o", str(d / "place")], check=True)

    def run(ring, recs, most, sizes):
        r = subprocess.run([str(d / "place")], input=f"{ring} {recs} {most} {len(sizes)} " + " ".join(map(str, sizes)),
                           capture_output=True, text=True, check=True)
        return [tuple(map(int, line.split())) for line in r.stdout.splitlines()]
    return run


@pytest.mark.parametrize("recs,ring,most", [(32, 224 * 1024, 64 * 1024), (16, 46 * 1024, 64 * 1024), (32, 4096, 1),
                                            (16, 4096, 10 ** 9)])
@pytest.mark.parametrize("kind", ["small", "large", "mixed", "one size"])
def test_placer(placer, recs, ring, most, kind):
    rng = random.Random(f"{recs} {kind} {most}")
    for _ in range(6):
        one = rng.randrange(1, ring // 128 + 1)
        top = ring // 128
        draw = {"small": lambda: rng.randrange(1, max(2, top // 20)), "large": lambda: rng.randrange(top // 3, top + 1),
                "mixed": lambda: rng.choice((1, 2, top // 7, top)), "one size": lambda: one}[kind]
        sizes = [128 * draw() for _ in range(rng.randrange(1, 200))]
        out = placer(ring, recs, most, sizes)
        assert len(out) == len(sizes)
        last_dep, end = -1, 0
        for j, (at, dep, land) in enumerate(out):
            assert at == (end if end + sizes[j] <= ring else 0)
            end = at + sizes[j]
            # done with: in order, the record's last chunk, and every chunk whose bytes are taken
            assert last_dep <= dep and j - recs <= dep < j
            for i in range(dep + 1, j):
                assert out[i][0] + sizes[i] <= at or end <= out[i][0]
            # ... and no more than that
            overlaps = [i for i in range(last_dep + 1, j) if out[i][0] < end and at < out[i][0] + sizes[i]]
            assert dep == max([last_dep, j - recs] + overlaps)
            last_dep = dep
            # landed: all but the fewest last chunks that hold `most` bytes, this one included
            fly, want = sizes[j], j - 1
            while want > dep and fly < most:
                fly += sizes[want]
                want -= 1
            assert land == want
