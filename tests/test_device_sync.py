"""What the CUDA sources say about memory order and convergence between threads,
checked as text: neither can be shown by running them."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "simplediffeq.jl_gb300", "csrc")


def code(name):
    """A source without its comments."""
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", " ", text, flags=re.S))


def test_parking_flags_are_released_and_acquired():
    """Every access to an entry's flag goes through flag_set (a release at GPU scope) or flag_seen (an acquire), and a
    __syncwarp carries what was acquired to the lanes that read the entries."""
    src = code("ode_solver.cuh")
    uses = re.findall(r"(\w+)\(ctl \+ PARK_FLAGS", src)
    assert sorted(uses) == ["flag_seen", "flag_set"] and src.count("PARK_FLAGS") == len(uses)
    assert re.search(r"flag_set\(int\* flag\) \{\s*asm volatile\(\"st\.release\.gpu\.", src)
    assert re.search(r"flag_seen\(const int\* flag\) \{\s*int v;\s*asm volatile\(\"ld\.acquire\.gpu\.", src)
    taken = src[src.index("flag_seen(ctl"):src.index("lane_unpark<PR, D, F, NK, KS, M::FSAL")]
    assert "__syncwarp()" in taken


def test_no_vote_over_the_threads_that_happen_to_be_there():
    """__activemask() names threads that nothing makes take part in the vote that follows it."""
    for path in glob.glob(os.path.join(CSRC, "*.cu*")) + glob.glob(os.path.join(CSRC, "*.h")):
        assert "__activemask" not in code(os.path.basename(path)), path
