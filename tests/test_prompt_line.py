"""Which prompts go to pairs of CTAs, from the library's own source: the order of a projection's sums hangs on it."""

import ctypes
import subprocess
from pathlib import Path

from megabake_b200.build import find_nvcc

SOURCE = Path(__file__).resolve().parent / "prompt_line.cu"


def test_prompts_of_up_to_128_tokens_are_summed_by_ctas_on_their_own(tmp_path):
    library = tmp_path / "line.so"
    subprocess.run([find_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17", "--extended-lambda", "-shared", "-Xcompiler",
                    "-fPIC", "-o", str(library), str(SOURCE)], check=True, capture_output=True, text=True)
    on_pairs = ctypes.CDLL(str(library)).on_pairs
    for sms in (148, 20, 2):
        assert not any(on_pairs(tokens, sms) for tokens in range(1, 129))
        assert all(on_pairs(tokens, sms) for tokens in (129, 256, 257, 512, 2048))
    assert not any(on_pairs(tokens, 1) for tokens in (1, 128, 129, 2048))
