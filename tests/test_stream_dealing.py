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


# us a step with three quarters of the SMs and with all of them, 16 layers (2: as said), a vocabulary of 49152:
# (batch, positions): (112 CTAs, 148 CTAs), taken in turn on one B200.  Two handles of the same plan are up to 3 % apart.
TIMES = {
    (576, 9, 3, 64, 1536, 16): {(1, 60): (249, 255), (8, 60): (264, 283), (1, 4000): (295, 304), (8, 4000): (318, 341), (1, 16000): (350, 348),
                                (8, 16000): (489, 518)},
    (576, 9, 3, 64, 1536, 2): {(1, 60): (55, 53), (8, 60): (60, 58), (8, 1000): (61, 58)},
    (896, 14, 2, 64, 4864, 16): {(1, 60): (300, 317), (8, 60): (325, 337), (1, 4000): (358, 386), (8, 4000): (370, 389)},
    (960, 15, 5, 64, 2560, 16): {(1, 60): (280, 298), (3, 1000): (297, 312), (3, 16000): (431, 442), (7, 2000): (338, 354), (8, 4000): (398, 394)},
    (1024, 16, 16, 64, 2816, 16): {(1, 60): (296, 303), (1, 16000): (431, 445), (2, 4000): (376, 365), (2, 16000): (645, 594), (3, 16000): (878, 753),
                                   (4, 4000): (468, 438), (8, 1000): (394, 363)},
    (1024, 16, 8, 128, 3072, 16): {(1, 60): (317, 326), (8, 1000): (428, 393), (8, 4000): (642, 628)},
    (1152, 18, 18, 64, 4608, 16): {(1, 60): (352, 333), (1, 4000): (396, 382), (4, 4000): (563, 510), (8, 60): (381, 359)},
    (1408, 22, 22, 64, 7168, 16): {(1, 60): (397, 402), (1, 4000): (441, 448), (3, 2000): (516, 477), (6, 2000): (589, 569), (8, 4000): (831, 853)},
    (768, 12, 12, 64, 3072, 16): {(1, 60): (281, 280), (4, 4000): (399, 368), (8, 60): (315, 302)},
    (512, 8, 8, 64, 1536, 16): {(1, 4000): (288, 312), (3, 1000): (271, 276), (4, 4000): (338, 332), (8, 60): (274, 286), (8, 4000): (439, 408)},
    (640, 10, 2, 64, 2560, 16): {(1, 60): (274, 282), (8, 60): (297, 312), (8, 4000): (339, 353)},
    (256, 4, 4, 64, 512, 8): {(1, 1000): (138, 134), (4, 1000): (142, 142), (4, 4000): (163, 153), (8, 4000): (179, 171)},
    (320, 5, 5, 64, 4992, 16): {(1, 300): (296, 301), (1, 16000): (390, 387), (4, 4000): (350, 353), (8, 4000): (408, 388)},
    (1536, 12, 2, 128, 8960, 16): {(1, 60): (491, 488), (8, 60): (537, 529)},
    (2048, 32, 32, 64, 8192, 16): {(1, 60): (544, 495), (4, 1000): (664, 585), (8, 4000): (1208, 1174)},
}


def _shape(sizes, sm_limit=0):
    hidden, heads, kv_heads, head_dim, intermediate, layers = sizes
    return (ctypes.c_int * 8)(hidden, heads, kv_heads, head_dim, intermediate, 49152, layers, sm_limit)


@pytest.mark.parametrize("sizes", TIMES)
def test_fewer_ctas_are_taken_where_they_were_measured_to_be_enough(deal, sizes):
    """No timed launch gets the slower number of CTAs by more than the scatter where fewer are taken, or by more than 5 % where all are."""
    chosen = set()
    for (batch, positions), (few, every) in TIMES[sizes].items():
        grid = deal.lib.grid_of(_shape(sizes), batch, 148)
        assert grid in (112, 148)
        assert few <= 1.03 * every if grid == 112 else every <= 1.05 * few, f"{sizes}: batch {batch}, {positions} positions"
        chosen.add(grid)
    if sizes[0] in (576, 896, 640) and sizes[5] == 16:
        assert chosen == {112}


def test_fewer_ctas_take_no_more_rounds_of_tiles(deal):
    """Over all shapes: where a launch has fewer CTAs, a layer's projections take no more rounds on the busiest CTA, summed up, than on
    all of them (a phase of its own may), and the output head a round a layer more at most; four CTAs to a sequence's KV head."""
    rng = random.Random(9)
    fewer = a_phase_more = 0
    for _ in range(6000):
        head_dim = rng.choice((64, 128))
        kv_heads = rng.randint(1, 16)
        heads = kv_heads * rng.randint(1, 8)
        sizes = (64 * rng.randint(6, 32), heads, kv_heads, head_dim, 64 * rng.randint(4, 140), rng.randint(1, 32))
        batch, sms = rng.randint(1, 32), rng.choice((148, 148, 132, 20))
        grid = deal.lib.grid_of(_shape(sizes), batch, sms)
        if grid == sms:
            continue
        fewer += 1
        assert batch <= 8 and sizes[0] >= 512 and grid >= 3 * sms // 4 and 4 * batch * kv_heads <= grid
        less, every = ([deal.lib.rounds_of(_shape(sizes), kind, n) for kind in range(5)] for n in (grid, sms))
        assert sum(less[:4]) <= sum(every[:4]) and less[4] <= every[4] + sizes[5]
        a_phase_more += any(a > b for a, b in zip(less[:4], every[:4]))
    assert fewer > 50 and a_phase_more > 0
    small = (576, 9, 3, 64, 1536, 30)
    assert deal.lib.grid_of(_shape(small, sm_limit=30), 1, 30) == 30 and deal.lib.grid_of(_shape(small), 1, 7) == 7
    assert deal.lib.grid_of(_shape(small), 9, 148) == deal.lib.grid_of(_shape(small), 17, 148) == 148


def test_quotients_of_the_probabilities_are_the_divisions(deal):
    """Every quotient is the division's while it and its remainder are normal numbers, and below that, of the smallest
    probabilities, after the rounding to bf16."""
    differ, rounded = ctypes.c_longlong(), ctypes.c_longlong()
    deal.lib.quotients(-80, 0, 4000000, ctypes.byref(differ), ctypes.byref(rounded))
    assert differ.value == 0 and rounded.value == 0
    deal.lib.quotients(-126, -81, 4000000, ctypes.byref(differ), ctypes.byref(rounded))
    assert rounded.value == 0
    deal.lib.quotient.restype = ctypes.c_float
    deal.lib.quotient.argtypes = [ctypes.c_float, ctypes.c_float]
    assert deal.lib.quotient(0.0, 3.0) == 0.0 and deal.lib.quotient(1.0, 1.0) == 1.0
    for a, b in ((float("nan"), 2.0), (1.0, float("nan")), (float("nan"), float("nan"))):
        assert deal.lib.quotient(a, b) != deal.lib.quotient(a, b)
