"""How the streaming decode kernel deals cached positions to CTAs, run on the host from the kernel's own source."""

import ctypes
import random
import subprocess
from pathlib import Path

import pytest

from megabake_b200.build import find_nvcc

SOURCE = Path(__file__).resolve().parent / "stream_dealing.cu"
LIST = 16  # parts a list of the kernel holds


@pytest.fixture(scope="module")
def deal(tmp_path_factory):
    library = tmp_path_factory.mktemp("dealing") / "dealing.so"
    subprocess.run([find_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                    "-o", str(library), str(SOURCE)], check=True, capture_output=True, text=True)
    lib = ctypes.CDLL(str(library))

    def run(lengths, heads=32, kv_heads=32, head_dim=64, batch=None, grid=148, ragged=True):
        longest, lists = ctypes.c_int(), ctypes.c_int()
        broken = lib.check_dealing(grid, batch or len(lengths), heads, kv_heads, head_dim, int(ragged), (ctypes.c_int * len(lengths))(*lengths),
                                   ctypes.byref(longest), ctypes.byref(lists))
        assert broken == 0, f"rule {broken} broken: lengths {lengths}, heads {heads}/{kv_heads} of {head_dim}, {grid} CTAs"
        return longest.value, lists.value

    run.lib = lib
    return run


# The parts of the busiest CTA, as these mixes were first seen to exceed one list of 16.
@pytest.mark.parametrize("lengths,parts", [([1000] * 28 + [10] * 4, 17), ([4000] * 9 + [10] * 7, 22), ([8000] * 6 + [10] * 6, 42)])
def test_long_sequences_beside_short_ones_need_several_lists(deal, lengths, parts):
    longest, lists = deal(lengths)
    assert longest == parts and lists == -(-parts // LIST)


def test_equal_lengths_need_one_list(deal):
    for batch in (1, 2, 7, 16, 32):
        for length in (0, 31, 255, 256, 1000, 2047, 16000):
            assert deal([length], batch=batch, ragged=False)[1] == 1


def test_every_position_is_dealt_exactly_once(deal):
    rng = random.Random(5)
    several = 0
    for _ in range(4000):
        heads, kv_heads, head_dim = rng.choice(((9, 3, 64), (14, 2, 64), (32, 32, 64), (32, 8, 128), (7, 1, 128), (16, 16, 128)))
        batch, grid, high = rng.randint(1, 32), rng.choice((148, 148, 132, 20, 3, 1)), rng.choice((40, 2048, 30000))
        few = rng.random()
        lengths = [rng.randint(0, high) if rng.random() < few else rng.randint(0, 60) for _ in range(batch)]
        several += deal(lengths, heads, kv_heads, head_dim, grid=grid)[1] > 1
        deal(lengths[:1], heads, kv_heads, head_dim, batch=batch, grid=grid, ragged=False)
    assert several > 100


@pytest.mark.parametrize("shape,fewer", [((576, 9, 3, 64, 1536), True), ((896, 14, 2, 64, 4864), True), ((2048, 32, 32, 64, 8192), False),
                                         ((320, 5, 5, 64, 4992), True)])
def test_fewer_ctas_only_where_no_phase_gets_longer(deal, shape, fewer):
    """135M, 0.5B and 1.7B shapes: three quarters of the SMs where that is no round of tiles more, for up to eight sequences."""
    grid = deal.lib.grid_of(*shape, 0, 0, 148)
    assert grid == (112 if fewer else 148)
    assert deal.lib.rounds_of(*shape, 0, grid) <= deal.lib.rounds_of(*shape, 0, 148)
    assert deal.lib.grid_of(*shape, 0, 1, 148) == deal.lib.grid_of(*shape, 0, 2, 148) == 148
    assert deal.lib.grid_of(*shape, 30, 0, 30) == 30 and deal.lib.grid_of(*shape, 0, 0, 7) == 7
