"""Which of its two kernels the prompt attention op takes, from the library's own source, against what both took on a B200."""

import ctypes
import subprocess
from pathlib import Path

import pytest

from megabake_b200.build import find_nvcc

SOURCE = Path(__file__).resolve().parent / "attention_line.cu"
# (head size, queries, keys, heads of all sequences, masked, us on tcgen05, us on mma.sync): graphs of twelve calls
MEASURED = [
    (64, 1, 65, 9, 1, 6.8, 6.3), (64, 1, 128, 9, 1, 6.8, 6.1), (64, 1, 512, 9, 1, 12.2, 13.1), (64, 16, 128, 9, 1, 6.8, 6.8), (64, 64, 65, 9, 1, 7.0, 7.8),
    (64, 64, 512, 9, 1, 12.4, 15.0), (64, 200, 200, 9, 1, 9.1, 9.7), (64, 192, 1024, 9, 1, 18.7, 25.2), (64, 64, 64, 9, 1, 6.2, 6.0),
    (64, 16, 16, 9, 1, 6.3, 5.2), (64, 129, 129, 9, 1, 9.5, 10.0), (64, 1, 65, 9, 0, 6.6, 5.7), (64, 1, 512, 9, 0, 11.9, 12.4), (64, 64, 128, 9, 0, 6.8, 6.9),
    (64, 320, 320, 9, 0, 9.8, 10.5), (64, 1, 65, 288, 1, 15.3, 8.5), (64, 64, 128, 288, 1, 14.7, 9.9), (64, 64, 512, 288, 1, 25.9, 21.6),
    (64, 65, 65, 288, 1, 15.2, 17.4), (64, 128, 128, 288, 1, 14.7, 18.4), (64, 320, 320, 288, 1, 58.0, 70.8), (64, 1, 512, 288, 0, 25.7, 16.8),
    (64, 129, 129, 288, 0, 33.6, 27.4), (64, 129, 512, 288, 0, 49.7, 50.7), (64, 320, 320, 56, 1, 19.0, 15.8), (64, 200, 200, 56, 1, 9.6, 13.7),
    (64, 320, 320, 56, 0, 19.4, 14.2), (64, 1, 128, 1024, 1, 48.1, 26.7), (64, 16, 512, 1024, 1, 92.3, 69.0), (64, 64, 128, 1024, 1, 49.9, 32.6),
    (64, 64, 512, 1024, 1, 95.4, 76.2), (64, 65, 65, 1024, 1, 50.5, 56.1), (64, 128, 512, 1024, 1, 90.9, 144.7), (64, 129, 129, 1024, 1, 123.6, 116.4),
    (64, 129, 512, 1024, 1, 174.3, 201.1), (64, 1, 65, 1024, 0, 48.6, 24.5), (64, 129, 129, 1024, 0, 115.1, 92.5), (64, 129, 512, 1024, 0, 178.7, 181.8),
    (64, 256, 256, 1024, 0, 131.8, 162.4), (64, 1, 128, 32, 1, 7.1, 6.2), (64, 128, 128, 32, 1, 7.1, 7.7), (64, 512, 512, 32, 1, 12.9, 21.4),
    (64, 1, 512, 128, 1, 13.4, 17.2), (64, 64, 1400, 128, 1, 24.5, 42.5), (64, 129, 129, 128, 0, 17.0, 17.9), (64, 1, 65, 448, 1, 26.1, 14.2),
    (64, 129, 129, 448, 0, 55.1, 43.1), (128, 1, 65, 32, 1, 8.8, 9.0), (128, 1, 128, 32, 0, 8.8, 8.8), (128, 1, 1400, 32, 1, 32.2, 41.6),
    (128, 16, 128, 32, 1, 8.3, 10.2), (128, 64, 64, 32, 1, 7.8, 9.3), (128, 128, 128, 32, 1, 9.2, 11.2), (128, 1, 128, 128, 1, 9.5, 9.1),
    (128, 1, 512, 128, 0, 17.0, 18.7), (128, 16, 128, 128, 0, 9.3, 10.2), (128, 65, 65, 128, 1, 9.6, 20.6), (128, 1, 128, 1024, 0, 60.7, 57.5),
    (128, 1, 512, 1024, 1, 129.7, 128.6), (128, 16, 512, 1024, 1, 130.4, 143.3), (128, 200, 200, 1024, 1, 176.4, 367.8), (64, 512, 512, 9, 1, 12.3, 15.6),
    (64, 320, 320, 64, 1, 19.4, 24.5), (64, 320, 320, 96, 1, 20.4, 29.3), (64, 256, 256, 56, 1, 9.5, 14.0), (64, 64, 128, 128, 1, 7.5, 9.4),
    (64, 64, 256, 128, 1, 9.5, 13.1), (64, 64, 320, 288, 1, 20.9, 15.9), (64, 64, 512, 448, 1, 49.3, 39.8), (64, 64, 1024, 288, 1, 38.6, 36.5),
    (64, 64, 1024, 1024, 1, 133.9, 125.8), (64, 16, 512, 288, 1, 25.8, 19.3), (64, 1, 256, 32, 1, 9.0, 8.6), (64, 1, 512, 288, 1, 26.7, 18.2),
    (64, 129, 128, 128, 1, 14.3, 16.4), (64, 129, 256, 448, 1, 58.1, 58.0), (64, 256, 256, 448, 1, 59.0, 80.2), (64, 160, 512, 288, 1, 49.0, 58.0),
    (64, 320, 512, 56, 1, 24.0, 21.6), (64, 320, 1024, 56, 1, 37.3, 36.2), (64, 300, 1400, 56, 1, 47.6, 45.0), (64, 1, 1400, 448, 1, 102.8, 80.5),
    (128, 1, 136, 32, 1, 10.7, 10.1), (128, 1, 512, 128, 1, 17.4, 19.1), (128, 1, 256, 1024, 1, 84.2, 82.8), (128, 1, 1400, 1024, 1, 293.4, 289.6),
    (128, 64, 128, 1024, 1, 64.7, 75.9)]
# Near the line: the fit is of times from before masks came in tiles.
NEAR = [
    (64, 129, 136, 288, 1, 34.1, 29.5), (64, 64, 512, 320, 1, 37.5, 33.2), (128, 8, 512, 128, 1, 16.6, 19.2), (128, 2, 512, 128, 1, 17.1, 19.3),
    (128, 4, 512, 128, 1, 16.8, 19.5)]


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    library = tmp_path_factory.mktemp("line") / "line.so"
    subprocess.run([find_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17", "--extended-lambda", "-shared", "-Xcompiler",
                    "-fPIC", "-o", str(library), str(SOURCE)], check=True, capture_output=True, text=True)
    loaded = ctypes.CDLL(str(library))
    chosen = loaded.on_tcgen05
    chosen.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_longlong, ctypes.c_int, ctypes.c_int, ctypes.c_int]
    chosen.library = loaded
    return chosen


@pytest.mark.parametrize("head_dim,queries,keys,heads,masked,tcgen05,mma", MEASURED)
def test_the_kernel_taken_is_the_faster_one_or_close(rule, head_dim, queries, keys, heads, masked, tcgen05, mma):
    """Within a tenth, what the fitted times are off by; a single tile stays with mma.sync whatever the head size."""
    taken, other = (tcgen05, mma) if rule(head_dim, queries, keys, heads, masked, 148, 0) else (mma, tcgen05)
    assert taken <= 1.1 * other or keys <= 64


@pytest.mark.parametrize("head_dim,queries,keys,heads,masked,tcgen05,mma", NEAR)
def test_near_the_line_the_kernel_taken_is_not_far_off(rule, head_dim, queries, keys, heads, masked, tcgen05, mma):
    """The largest misses over 423 shapes, all within a fifth."""
    taken, other = (tcgen05, mma) if rule(head_dim, queries, keys, heads, masked, 148, 0) else (mma, tcgen05)
    assert taken <= 1.2 * other


def test_sizes_at_the_ends_of_the_range_are_taken(rule):
    for head_dim in (64, 128):
        for queries, keys, heads in ((1, 1, 1), (1, 10240, 1), (2**31 - 1, 2**31 - 1, 2**31), (1, 65, 2**40)):
            for sms, limited in ((148, 0), (1, 1)):
                assert rule(head_dim, queries, keys, heads, 0, sms, limited) in (0, 1)


# (head size, heads, sequences, queries, keys, us with plain loads, us with tiled copies) of the tcgen05 kernel, masks on 16-byte rows
MASKS = [
    (64, 32, 4, 1, 128, 7.9, 9.9), (64, 32, 4, 1, 512, 13.6, 20.6), (64, 32, 9, 1, 1400, 54.5, 62.9), (64, 32, 32, 1, 512, 91.5, 116.0),
    (64, 32, 1, 16, 72, 7.0, 7.3), (64, 32, 4, 16, 640, 15.1, 17.4), (64, 32, 4, 24, 128, 7.5, 8.9), (64, 32, 4, 24, 512, 13.3, 14.2),
    (64, 32, 4, 16, 1024, 20.6, 19.6), (64, 9, 1, 24, 2048, 34.4, 31.5), (64, 32, 4, 65, 200, 9.8, 10.8), (64, 32, 4, 65, 1024, 20.9, 19.7),
    (64, 32, 4, 96, 128, 7.8, 7.7), (64, 32, 4, 128, 72, 8.2, 8.5), (64, 32, 1, 128, 512, 13.5, 12.3), (64, 9, 1, 200, 896, 19.1, 17.1),
    (64, 32, 4, 1024, 1152, 163.0, 145.2), (128, 32, 4, 1, 512, 17.4, 22.1), (128, 32, 1, 16, 2048, 43.2, 45.7), (128, 32, 4, 65, 72, 9.7, 10.6),
    (128, 32, 1, 64, 1400, 33.4, 34.4), (128, 32, 1, 96, 72, 8.9, 9.2), (128, 32, 1, 96, 256, 12.1, 11.6), (128, 32, 4, 128, 72, 10.1, 11.1),
    (128, 32, 1, 200, 200, 12.6, 12.6), (128, 32, 1, 200, 2048, 50.2, 46.1), (128, 32, 1, 512, 512, 20.3, 18.1), (128, 32, 4, 200, 640, 42.3, 39.2),
    (128, 32, 4, 1024, 72, 65.3, 67.6), (128, 9, 1, 65, 2048, 45.0, 44.8)]


@pytest.mark.parametrize("head_dim,heads,batch,queries,keys,loads,tiles", MASKS)
def test_a_mask_comes_the_faster_way_or_close(rule, head_dim, heads, batch, queries, keys, loads, tiles):
    """Or within 6 %, where the rule's lines cross what was measured."""
    taken, other = (tiles, loads) if rule.library.mask_in_tiles(head_dim, queries, keys) else (loads, tiles)
    assert taken <= 1.06 * other


# The same of masks whose rows begin off 16-byte boundaries, and copies of every eighth row
EIGHTHS = [
    (64, 32, 1, 96, 130, 8.7, 8.1), (64, 32, 1, 130, 75, 7.8, 8.4), (64, 32, 1, 130, 205, 11.2, 12.1), (64, 32, 1, 130, 330, 15.2, 14.5),
    (64, 32, 1, 200, 75, 7.8, 8.0), (64, 32, 1, 200, 205, 11.2, 9.5), (64, 32, 1, 500, 130, 9.8, 9.3), (64, 32, 1, 500, 1030, 30.5, 22.0),
    (64, 32, 4, 16, 650, 17.6, 24.7), (64, 32, 4, 16, 1030, 24.1, 26.8), (64, 32, 4, 32, 330, 12.1, 16.4), (64, 32, 4, 32, 650, 18.3, 16.6),
    (64, 32, 4, 64, 205, 10.3, 11.2), (64, 32, 4, 64, 330, 13.0, 11.9), (64, 32, 4, 96, 130, 9.4, 9.4), (64, 9, 1, 500, 650, 23.1, 15.1),
    (64, 9, 4, 32, 75, 6.7, 7.5), (64, 9, 4, 200, 330, 15.2, 10.9), (128, 32, 1, 16, 1030, 27.5, 30.4), (128, 32, 1, 96, 205, 12.4, 11.6),
    (128, 32, 1, 130, 205, 13.4, 13.9), (128, 32, 1, 200, 330, 18.4, 15.4), (128, 32, 1, 500, 75, 9.9, 10.7), (128, 32, 1, 500, 650, 29.2, 23.8),
    (128, 32, 4, 32, 650, 22.1, 23.8), (128, 32, 4, 64, 205, 12.5, 13.3), (128, 32, 4, 130, 330, 32.7, 31.0), (128, 32, 4, 200, 1030, 68.4, 66.0)]


@pytest.mark.parametrize("head_dim,heads,batch,queries,keys,loads,copies", EIGHTHS)
def test_a_mask_off_16_bytes_comes_the_faster_way_or_close(rule, head_dim, heads, batch, queries, keys, loads, copies):
    taken, other = (copies, loads) if rule.library.mask_in_eights(head_dim, queries, keys) else (loads, copies)
    assert taken <= 1.06 * other
