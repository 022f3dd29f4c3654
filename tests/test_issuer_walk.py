"""The K blocks of the kernel's MMA-issuing threads, from the header that the kernel includes: every block has one issuer and the
ring position of its number, and every ring stage has one issuer, in odd rings too. (A barrier wait tells only a phase's parity,
so an issuer that did not see the use before must not wait on a stage: its wait can pass while that use is outstanding.)"""
import os
import random
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "amd_developer_challenge_2025_b200", "csrc")
PROGRAM = """
#include <cstdio>
#include <cstdlib>
#include "issuer_walk.h"
// walk <me> <issuers> <stages> <buffers> <blocks of tile 0> <blocks of tile 1> ...: "block stage phase buffer" of each issue
int main(int argc, char** argv) {
  const int me = atoi(argv[1]), issuers = atoi(argv[2]), stages = atoi(argv[3]), buffers = atoi(argv[4]);
  IssuerWalk at;
  at.begin(me, stages, buffers);
  int base = 0;
  for (int t = 5; t < argc; ++t) {
    const int blocks = atoi(argv[t]);
    while (at.block < blocks) {
      printf("%d %d %u %d\\n", base + at.block, at.stage, at.phase, at.buffer);
      at.next(me, issuers, stages, buffers);
    }
    at.block -= blocks;
    base += blocks;
  }
}
"""


@pytest.fixture(scope="module")
def walk(tmp_path_factory):
    cxx = os.environ.get("CXX") or shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("walk")
    (d / "walk.cpp").write_text(PROGRAM)
    subprocess.check_call([cxx, "-std=c++17", f"-I{CSRC}", str(d / "walk.cpp"), "-o", str(d / "walk")])
    return lambda *args: [tuple(map(int, line.split())) for line in
                          subprocess.check_output([str(d / "walk"), *map(str, args)], text=True).splitlines()]


@pytest.mark.parametrize("stages", range(2, 9))
@pytest.mark.parametrize("issuers", [1, 2])
@pytest.mark.parametrize("most_buffers", [2, 4])
def test_every_stage_has_one_issuer(walk, stages, issuers, most_buffers):
    buffers = min(most_buffers, stages)
    rng = random.Random(10 * stages + issuers)
    for tiles in ([57], [1] * 40, [rng.randint(1, 9) for _ in range(30)]):
        owner, seen = {}, []
        for me in range(issuers):
            mine = walk(me, issuers, stages, buffers, *tiles)
            assert [j for j, *_ in mine] == sorted(j for j, *_ in mine)
            for j, stage, phase, buffer in mine:
                assert (stage, phase, buffer) == (j % stages, (j // stages) % 2, j % buffers)
                assert owner.setdefault(stage, me) == me
            seen += [j for j, *_ in mine]
        assert sorted(seen) == list(range(sum(tiles)))
