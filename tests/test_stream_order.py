"""What a CTA of the streaming decode kernel has read when it looks for another's results, on the host from the kernel's own source."""

import ctypes
import random
import subprocess
from pathlib import Path

import pytest

from megabake_b200.build import find_nvcc

SOURCE = Path(__file__).resolve().parent / "stream_order.cu"


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    library = tmp_path_factory.mktemp("order") / "order.so"
    subprocess.run([find_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                    "-o", str(library), str(SOURCE)], check=True, capture_output=True, text=True)
    return ctypes.CDLL(str(library))


def _shape(hidden, heads, kv_heads, head_dim, intermediate, layers=8, vocab=49152, sm_limit=0):
    return (ctypes.c_int * 8)(hidden, heads, kv_heads, head_dim, intermediate, vocab, layers, sm_limit)


def _shapes(count, seed):
    """Small shapes, where units are few, among all that the kernel takes."""
    rng = random.Random(seed)
    while count > 0:
        head_dim, kv_heads = rng.choice((64, 128)), rng.randint(1, 4) if rng.random() < 0.7 else rng.randint(5, 32)
        small = rng.random() < 0.6
        sizes = (64 * (rng.randint(1, 6) if small else rng.randint(7, 32)), kv_heads * rng.randint(1, 8), kv_heads, head_dim,
                 64 * (rng.randint(1, 12) if small else rng.randint(4, 140)))
        if sizes[1] <= 64:
            count -= 1
            yield sizes, rng.randint(1, 32), rng.choice((148, 148, 132, 20, 3, 2))


def test_every_cta_of_the_output_head_has_a_unit_of_each_layer(lib):
    ctas = ctypes.c_int()
    fewer = 0
    for sizes, batch, sms in [((128, 2, 1, 64, 256), 1, 148), ((128, 2, 2, 64, 256), 16, 148), ((64, 1, 1, 64, 64), 32, 148), *_shapes(4000, 3)]:
        if lib.has_plan(_shape(*sizes)):
            idle = lib.ctas_without_a_layer(_shape(*sizes), batch, sms, ctypes.byref(ctas))
            assert idle == 0, f"{sizes}, {batch} sequences, {sms} SMs: {idle} of {ctas.value} CTAs"
            fewer += ctas.value < sms and sizes[0] < 512
    assert fewer > 50
    for sizes in ((576, 9, 3, 64, 1536), (896, 14, 2, 64, 4864), (2048, 32, 32, 64, 8192)):
        lib.ctas_without_a_layer(_shape(*sizes), 16, 148, ctypes.byref(ctas))
        assert ctas.value == 148


DOWN, HEAD = 3, 4
MODELS = ((576, 9, 3, 64, 1536), (896, 14, 2, 64, 4864), (2048, 32, 32, 64, 8192))


def _early(lib, sizes, batch, sms, lengths, met):
    where = (ctypes.c_int * 4)(-1, -1, -1, -1)
    found = lib.looks_too_early(_shape(*sizes), batch, sms, int(len(lengths) > 1), (ctypes.c_int * len(lengths))(*lengths), met, where)
    return found, f"{sizes}, {batch} sequences, {sms} SMs, {lengths}: {found}, CTA {where[0]} of {where[1]} in layer {where[2]}, step {where[3]}"


def test_no_cta_looks_for_a_word_before_it_knows_of_its_reset(lib):
    """Buffers are used in turn by three layers.  Whoever looks for a word must depend on something its last writer stored behind a fence
    behind the reset of what was there, or it may take that."""
    assert lib.fence_met() == DOWN
    cases = [(sizes, batch, 148, [length]) for sizes in MODELS for batch in (1, 3, 8, 16, 32) for length in (0, 1000)]
    cases += [((256, 4, 2, 64, 512), 1, 148, [5]), ((256, 4, 4, 64, 512), 16, 148, [300])]
    rng = random.Random(7)
    for sizes, batch, sms in _shapes(60, 5):
        cases += [(sizes, batch, sms, [rng.randint(0, 600)]), (sizes, batch, sms, [rng.randint(0, 3000) if rng.random() < 0.3 else 9 for _ in range(batch)])]
    for sizes, batch, sms, lengths in cases:
        if lib.has_plan(_shape(*sizes)):
            found, what = _early(lib, sizes, batch, sms, lengths, lib.fence_met())
            assert found == 0, what


def test_a_fence_behind_down_proj_would_be_too_late(lib):
    """The same walk sees it in small shapes; in the models' every CTA has other work that comes behind the fence."""
    assert _early(lib, (256, 4, 2, 64, 512), 1, 148, [5], HEAD)[0] > 0
    for sizes in MODELS:
        for batch in (1, 3, 8, 12, 16, 32):
            assert _early(lib, sizes, batch, 148, [1000], HEAD)[0] == 0
