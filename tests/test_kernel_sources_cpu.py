"""Rules of the kernels that reading the sources can check."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "dft-efe_gb300" / "csrc"
SOURCES = sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh"))


def code(path):
    return re.sub(r"//[^\n]*", "", path.read_text())


def tmem_kernels():
    """(name, body) of every kernel that allocates TMEM."""
    for path in SOURCES:
        parts = re.split(r"\b__global__\b", code(path))[1:]
        for part in parts:
            body = part.split("\n}\n", 1)[0]
            if "tcgen05.alloc" in body:
                yield re.search(r"\b(k_\w+)\s*\(", body).group(1), body


KERNELS = dict(tmem_kernels())


def test_kernels_found():
    assert {"k_cell_apply_tc2", "k_cell_apply_oz", "k_cell_apply_shared", "k_oz_gram", "k_oz_rot"} <= set(KERNELS)


@pytest.mark.parametrize("name", sorted(KERNELS))
def test_successor_is_released_after_the_tmem_allocation(name):
    """A successor with early launch may own TMEM while it waits for this kernel: it must not become resident before
    every block of this kernel owns its columns (allocation, then the barrier that publishes it, then the trigger)."""
    body = KERNELS[name]
    assert "pdl_enter" not in body
    at = body.find("pdl_trigger(")
    if at >= 0:
        alloc = body.find("tcgen05.alloc")
        barrier = body.find("__syncthreads()", alloc)
        assert alloc < barrier < at


def test_fork_of_the_size_groups_follows_the_folded_tiles():
    """The side stream's size group waits for the fork event alone, so the event is recorded after the tiles are
    built."""
    src = code(CSRC / "gbfe_core.cu")
    body = src[src.index("bool filter_step_fused("):]
    body = body[:body.index("\n}\n")]
    assert 0 <= body.index("build_tc_mats_folded(") < body.index("cudaEventRecord(ctx->fork_ev")


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_no_copy_to_several_blocks(path):
    """The library also serves several processes on several GPUs, where every block copies its own tiles."""
    assert "multicast" not in code(path)
