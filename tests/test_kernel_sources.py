"""What the kernels must not leave to chance and a run on a GPU need not show,
read off the sources (single-svdlib_b200/csrc)."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "single-svdlib_b200", "csrc")


def source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


def test_resident_lanczos_waits_for_its_cluster_before_the_first_remote_store():
    """A CTA may touch another's shared memory only once that one has started."""
    text = source("lanczos_kernel.cu")
    body = text[text.index("k_lanczos_block(const __grid_constant__ LzArgs a)"):]
    before = body[:body.index("while (j < a.last)")]
    assert "map_shared_rank" not in before
    assert "cg::this_cluster().sync();" in before


def test_dynamic_shared_memory_is_aligned_as_it_is_used():
    """Dynamic shared memory that is read and written 16 bytes at a time asks for
    that alignment (dense_split.cu aligns its own base)."""
    seen = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = source(os.path.basename(path))
        for decl in re.findall(r"extern __shared__[^;]*;", text):
            if os.path.basename(path) == "dense_split.cu":
                continue
            seen += 1
            m = re.search(r"__align__\((\d+)\)", decl)
            assert m and int(m.group(1)) >= 16, (os.path.basename(path), decl)
    assert seen >= 15
