"""A prompt projection's CTA leaves when every use of its pipeline has been consumed, run on the host from the kernel's own source."""

import ctypes
import subprocess
from pathlib import Path

from megabake_b200.build import find_nvcc

SOURCE = Path(__file__).resolve().parent / "prompt_drain.cu"


def test_no_cta_leaves_before_its_last_use_is_consumed(tmp_path):
    library = tmp_path / "drain.so"
    subprocess.run([find_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17", "--extended-lambda", "-shared", "-Xcompiler",
                    "-fPIC", "-o", str(library), str(SOURCE)], check=True, capture_output=True, text=True)
    left = ctypes.CDLL(str(library)).uses_consumed_when_left
    for stages in range(2, 17):
        for uses in range(0, 5 * stages + 3):  # fewer uses than slots among them: one short unit to a CTA
            assert left(uses, stages) == uses, (stages, uses)
