"""The words of shared memory by which the tensor engine's workers tell its producers that operands are complete: a producer's copies read
what other CTAs have stored, which the worker that waited for them has acquired, so the word has to release and acquire in turn."""

import re
from pathlib import Path

SOURCES = sorted((Path(__file__).resolve().parent.parent / "megabake_b200" / "csrc").glob("*.cu*"))


def test_ready_words_are_released_and_acquired():
    uses = {"b_ready": [], "a_ready": []}
    for source in SOURCES:
        for line in source.read_text().splitlines():
            code = line.split("//")[0]
            for name in uses:
                if re.search(rf"\b{name}\b", code):
                    uses[name].append(code.strip())
    for name, lines in uses.items():
        stores = [line for line in lines if f"st_release_shared_s32(&cx.tc->{name}," in line]
        loads = [line for line in lines if re.search(rf"ld_acquire_shared_s32\(&(cx\.)?tc->{name}\)", line)]
        rest = [line for line in lines if line not in stores and line not in loads]
        assert stores and loads
        # the declaration, and the value it has before the CTA's first block barrier
        assert all(re.fullmatch(rf"int {name};|cx\.tc->{name} = 0;", line) for line in rest), rest
