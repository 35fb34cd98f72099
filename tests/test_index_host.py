"""Offsets of the C-PML memory variables are formed in 64 bits.  A slab holds
fewer than 2^31 cells, six of them more: on an 85 x 2500 x 2500 grid with 40
absorbing cells (5.3e8 cells, 64 GB of state, accepted) the last z variable
starts 5 * 5e8 elements in."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "efwi-3d_b200", "csrc")
SOURCES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h")))


def test_offsets_of_a_large_slab_need_64_bits():
    nz, nx, ny, npml = 85, 2500, 2500, 40
    slab = 2 * npml * nx * ny
    assert nz * nx * ny < 2 ** 31 and slab < 2 ** 31 and 5 * slab >= 2 ** 31


@pytest.mark.parametrize("name", SOURCES)
def test_no_kernel_narrows_a_slab_size(name):
    src = open(os.path.join(CSRC, name)).read()
    src = re.sub(r"//[^\n]*|/\*.*?\*/", "", src, flags=re.S)
    # casts, and int variables initialised from one
    bad = re.findall(r"\(int\)\s*[\w.>-]*\bslab_[zxy]\b", src)
    for decl in re.findall(r"(?<!long )\b(?:int|unsigned|uint32_t|int32_t)\s+(\w+\s*=[^;{}]*);", src):
        bad += re.findall(r"\w+\s*=\s*(?:[\w.>-]*\.)?slab_[zxy]\b", decl)
    assert not bad
    if name == "efwi_common.cuh":
        assert re.search(r"long long slab_z, slab_x, slab_y;", src)
