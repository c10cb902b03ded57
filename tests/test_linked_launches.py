"""Rules that the kernels of a step or a sort keep, since a linked kernel is
resident before the writes of the kernel ahead of it are visible. They are
checked in the source: what a wrong load reads on a GPU depends on timing."""

import re

import pytest

from conftest import PKG

CSRC = PKG / "csrc"
LINKED = ["grid_sort.cu", "grid_sort.cuh", "world.cu", "world_contacts.cuh", "world_kernels.cuh", "world_slots.cuh",
          "world_tiles.cuh"]

# What is made at build, or copied to the device between steps, and written by
# no kernel: chunk lists, primitives (as words, and their planes), SDF voxels,
# and the members of shape-matching clusters.
TABLES = {
    "world_kernels.cuh": {"list": "chunk_slot", "b": "sdf_trilinear", "V.plane4": None},
    "world.cu": {"w": "stage_prims", "V.mem_info": None, "V.mem": None, "V.mem_soft": None},
}


def source(name):
    text = (CSRC / name).read_text()
    return re.sub(r"//[^\n]*", "", text)


@pytest.mark.parametrize("name", LINKED)
def test_read_only_loads_are_of_build_time_tables(name):
    """__ldg and ld.global.nc need data that nobody writes while the kernel
    lives: not what an earlier kernel of the same step writes."""
    text = source(name)
    assert "ld.global.nc" not in text
    for m in re.finditer(r"__ldg\(\s*([\w.]+)", text):
        tables = TABLES.get(name, {})
        assert m.group(1) in tables, f"{name}: __ldg of {m.group(1)}"
        # short names stand for a table in one function only
        fn = tables[m.group(1)]
        if fn:
            heads = re.findall(r"__forceinline__[^;{]*?(\w+)\(", text[: m.start()])
            assert heads[-1] == fn, f"{name}: __ldg of {m.group(1)} in {heads[-1]}"


@pytest.mark.parametrize("name", LINKED)
def test_kernels_wait_before_anything_else(name):
    """Every kernel starts with pdl_begin(); only the cloth's colours, which
    look up what no kernel just ahead of them writes, may have it later."""
    bodies = re.findall(r"__global__[^;{]*?\b(k_\w+)\(([^;{]*)\)\s*\{\s*([^;]*;)", source(name))
    for kernel, _, first in bodies:
        want = "if (!early) pdl_begin();" if kernel in ("k_cloth", "k_bend", "k_tether") else "pdl_begin();"
        assert first.strip() == want, f"{name}: {kernel} starts with {first.strip()}"
