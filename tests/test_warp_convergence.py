"""Instructions that every lane of a warp has to execute together (the .aligned forms of the
cluster barriers and of the tensor-memory instructions, votes over a mask) stand where the
lanes are known to be together: read from the kernels' source, since a compiler that happens to
reconverge a warp hides the fault on the GPU."""
import glob
import os
import re

from conftest import PKG


def sources():
    for path in sorted(glob.glob(os.path.join(PKG, "csrc", "*.cu*"))):
        text = open(path).read()
        yield os.path.basename(path), re.sub(r"//[^\n]*", "", text)


def test_no_vote_over_the_lanes_that_happen_to_be_active():
    for name, text in sources():
        assert "__activemask" not in text, name


def test_aligned_warp_instructions_follow_a_convergence_point():
    found = 0
    for name, text in sources():
        if name != "field_tm.cuh":
            continue
        lines = [l.strip() for l in text.split("\n") if l.strip()]
        for i, line in enumerate(lines):
            if not re.search(r'"(barrier\.cluster|tcgen05)\.[a-z0-9_:.]*aligned', line):
                continue
            found += 1
            # back to the statement before this one, over the asm's own lines, the warp's own
            # uniform branch and declarations; the warp-wide instruction before it may be one of these
            j, ok = i - 1, False
            while j >= 0 and i - j < 12:
                if re.search(r"__sync(warp|threads)\(|\.aligned", lines[j]):
                    ok = True
                    break
                if not re.match(r'(asm volatile\($|"|if constexpr|if \(warp == 0\)|const uint32_t sadr|uint32_t r\[16\]|'
                                r'__device__ __forceinline__ void tm_|\}? ?else|\{|:)', lines[j]):
                    break
                if lines[j].startswith("__device__"):  # tm_put8, tm_get8: their callers converge first
                    calls = [k for k, l in enumerate(lines) if re.search(r"\btm_(put|get)8\(tm", l)]
                    ok = all("__syncwarp();" in lines[k - 1] for k in calls) and len(calls) >= 2
                    break
                j -= 1
            assert ok, (name, line, lines[max(j, 0)])
    assert found >= 8
