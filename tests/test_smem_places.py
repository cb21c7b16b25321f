"""The shared-memory requests that set how many blocks an SM holds
(csrc/places.h), as host code: exactly as many places as asked for."""
from __future__ import annotations

import os
import subprocess

import pytest

from conftest import PKG

# per SM, reserved per block, most per block, in bytes
LIMITS = [(233472, 1024, 232448), (167936, 1024, 166912)]

PROGRAM = """
#include <cstdio>
#include "places.h"
int main() {
    unsigned long per_sm, reserved, per_block, smem;
    unsigned places;
    while (std::scanf("%lu %lu %lu %lu %u", &per_sm, &reserved, &per_block, &smem, &places) == 5) {
        const mi::SmemLimits L{per_sm, reserved, per_block};
        std::printf("%lu %u\\n", (unsigned long)mi::smem_for_places(L, smem, places), mi::smem_places(L, smem));
    }
}
"""


@pytest.fixture(scope="module")
def places(tmp_path_factory):
    d = tmp_path_factory.mktemp("places")
    (d / "main.cpp").write_text(PROGRAM)
    exe = str(d / "main")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(PKG, "csrc"), str(d / "main.cpp"),
                    "-o", exe], check=True)

    def run(rows):
        text = "\n".join(" ".join(map(str, r)) for r in rows)
        out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout
        return [tuple(map(int, line.split())) for line in out.splitlines()]

    return run


@pytest.mark.parametrize("limits", LIMITS)
def test_request_holds_the_places_and_no_more(places, limits):
    per_sm, reserved, per_block = limits
    for want in range(1, 25):
        small = [limits + (smem, want) for smem in (0, 1, 128, 4096, 7000)]
        for (got, _), (_, _, _, smem, _) in zip(places(small), small):
            assert smem <= got <= per_block
            block = -(-(got + reserved) // 128) * 128
            held = per_sm // block
            if got > smem:      # the request was raised: the places, exactly
                assert held == want or (got == per_block and held < want), (want, smem, got)
            else:               # the kernel's own need already limits it
                assert held <= want, (want, smem, got)


def test_a_request_is_never_lowered(places):
    big = [LIMITS[0] + (smem, n) for smem in (20000, 60000, 120000, 232448) for n in (1, 2, 4, 12, 16)]
    assert all(got >= row[3] for (got, _), row in zip(places(big), big))
