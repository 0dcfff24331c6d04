"""Which of its two kernels the prompt attention op takes, from the library's own source, against what both took on a B200."""

import ctypes
import subprocess
from pathlib import Path

import pytest

from megabake_b200.build import find_nvcc

SOURCE = Path(__file__).resolve().parent / "attention_line.cu"
# (head size, queries, keys, heads of all sequences, masked, us on tcgen05, us on mma.sync): graphs of twelve calls
MEASURED = [
    (64, 1, 65, 9, 1, 6.8, 6.8), (64, 1, 128, 9, 1, 7.0, 6.3), (64, 1, 512, 9, 1, 12.4, 13.7), (64, 16, 128, 9, 1, 7.0, 7.0), (64, 64, 65, 9, 1, 7.0, 8.1),
    (64, 64, 512, 9, 1, 12.4, 15.3), (64, 200, 200, 9, 1, 9.8, 9.9), (64, 192, 1024, 9, 1, 20.5, 25.7), (64, 64, 64, 9, 1, 6.2, 6.2), (64, 16, 16, 9, 1, 6.4, 5.5),
    (64, 129, 129, 9, 1, 9.3, 10.8), (64, 1, 65, 9, 0, 6.8, 5.7), (64, 1, 512, 9, 0, 12.1, 12.2), (64, 64, 128, 9, 0, 6.9, 7.0), (64, 320, 320, 9, 0, 9.9, 10.5),
    (64, 1, 65, 288, 1, 15.5, 9.0), (64, 64, 128, 288, 1, 15.9, 11.3), (64, 64, 512, 288, 1, 27.5, 23.0), (64, 65, 65, 288, 1, 15.9, 18.9), (64, 128, 128, 288, 1, 16.9, 21.1),
    (64, 320, 320, 288, 1, 65.5, 75.7), (64, 1, 512, 288, 0, 26.9, 17.8), (64, 129, 129, 288, 0, 35.4, 30.3), (64, 129, 512, 288, 0, 51.6, 53.3), (64, 320, 320, 56, 1, 20.6, 16.1),
    (64, 200, 200, 56, 1, 10.2, 16.5), (64, 320, 320, 56, 0, 19.1, 14.6), (64, 1, 128, 1024, 1, 52.5, 30.9), (64, 16, 512, 1024, 1, 92.8, 70.8), (64, 64, 128, 1024, 1, 54.8, 37.4),
    (64, 64, 512, 1024, 1, 95.1, 77.9), (64, 65, 65, 1024, 1, 54.7, 66.4), (64, 128, 512, 1024, 1, 100.2, 146.2), (64, 129, 129, 1024, 1, 127.3, 131.0), (64, 129, 512, 1024, 1, 186.7, 203.7),
    (64, 1, 65, 1024, 0, 53.1, 28.1), (64, 129, 129, 1024, 0, 120.8, 100.9), (64, 129, 512, 1024, 0, 178.3, 182.0), (64, 256, 256, 1024, 0, 130.4, 164.4), (64, 1, 128, 32, 1, 7.2, 6.5),
    (64, 128, 128, 32, 1, 7.5, 8.2), (64, 512, 512, 32, 1, 14.3, 21.6), (64, 1, 512, 128, 1, 14.8, 18.4), (64, 64, 1400, 128, 1, 28.2, 43.9), (64, 129, 129, 128, 0, 18.3, 19.2),
    (64, 1, 65, 448, 1, 25.4, 16.2), (64, 129, 129, 448, 0, 57.0, 48.3), (128, 1, 65, 32, 1, 9.2, 9.9), (128, 1, 128, 32, 0, 9.2, 8.7), (128, 1, 1400, 32, 1, 38.0, 42.5),
    (128, 16, 128, 32, 1, 9.0, 10.2), (128, 64, 64, 32, 1, 8.3, 9.4), (128, 128, 128, 32, 1, 9.6, 11.3), (128, 1, 128, 128, 1, 10.2, 9.3), (128, 1, 512, 128, 0, 19.6, 18.8),
    (128, 16, 128, 128, 0, 10.1, 10.3), (128, 65, 65, 128, 1, 10.2, 22.7), (128, 1, 128, 1024, 0, 66.5, 57.7), (128, 1, 512, 1024, 1, 127.5, 129.2), (128, 16, 512, 1024, 1, 128.3, 142.8),
    (128, 200, 200, 1024, 1, 178.0, 361.7)]


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
