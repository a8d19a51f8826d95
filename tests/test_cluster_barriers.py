"""Every aligned cluster barrier in the kernel sources is reached by converged
warps: the statement before it is a warp or block barrier (or the other half of
the same cluster barrier).  Warps that arrive divergently can hang the GPU, so
the rule is checked on the sources."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "parareal-cc-cfv-split-gpu_b200" / "csrc"
ALIGNED = re.compile(r"barrier\.cluster\.(arrive|wait)[.\w]*\.aligned")
CONVERGED = re.compile(r"__sync(warp|threads)\(|barrier\.cluster\.")


def _statements(text):
    """Source lines without comments and blank lines."""
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    lines = [re.sub(r"//.*", "", ln).strip() for ln in text.splitlines()]
    return [ln for ln in lines if ln]


def unguarded(text):
    st = _statements(text)
    return [ln for prev, ln in zip([""] + st, st) if ALIGNED.search(ln) and not CONVERGED.search(prev)]


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cu")), ids=lambda p: p.name)
def test_aligned_cluster_barriers_follow_a_warp_barrier(path):
    assert unguarded(path.read_text()) == []


def test_the_check_sees_an_unguarded_barrier():
    bad = 'if (threadIdx.x < 5) a[0] = 1;\nasm volatile("barrier.cluster.arrive.aligned;");\n'
    assert len(unguarded(bad)) == 1
    assert unguarded(bad.replace("= 1;\n", "= 1;\n__syncwarp();\n// why\n")) == []
