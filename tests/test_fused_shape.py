"""Which 1x1 pairs are fused (katago_b200/csrc/kb_fused_shape.h, compiled here; no GPU needed): in every shape that is, each wait of
the first epilogue names the part it means.  A wait is by parity; it passes while its barrier is in a phase of the other parity, so
a warp must know of all of the accumulator's turns but the last."""
import ctypes
import os
import subprocess

import pytest

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_WARPS = 3  # per lane quarter


@pytest.fixture(scope="module")
def shape(tmp_path_factory):
    d = tmp_path_factory.mktemp("fused_shape")
    (d / "s.cpp").write_text('#include "kb_fused_shape.h"\nextern "C" int parts(int ct, int cn) { return kb::postPrePartWidth(ct, cn); }\n'
                             'extern "C" int accumulators(int np, int cn) { return kb::postPreAccumulators(np, cn); }\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(_ROOT, "katago_b200", "csrc"), "-o", str(d / "s.so"), str(d / "s.cpp")], check=True)
    return ctypes.CDLL(str(d / "s.so"))


def _passes_early(ct, np_, accumulators):
    """(warp, part) of the waits that can pass before their part is done."""
    units, per_part, parts = ct // 32, np_ // 32, ct // np_
    found = []
    for cg in range(_WARPS):
        known = -1  # parts up to this one are done: they complete in order
        for part in (t * parts + u // per_part for t in range(5) for u in range(cg, units, _WARPS)):
            turn, done = part // accumulators, len([p for p in range(known + 1) if p % accumulators == part % accumulators])
            # phases that may be complete by now: `done` or more; a wait for `turn` passes where the last complete one has its parity
            found += [(cg, part) for last in range(done - 1, turn) if (last - turn) % 2 == 0]
            known = max(known, part)
    return found


def test_a_warp_that_skips_two_parts_is_found():
    assert _passes_early(448, 64, 2) and not _passes_early(320, 64, 2) and not _passes_early(448, 224, 1)


@pytest.mark.parametrize("cn", range(64, 257, 32))
def test_waits_of_the_first_epilogue_name_their_part(cn, shape):
    fused = 0
    for ct in range(64, 2049, 64):
        np_ = shape.parts(ct, cn)
        if np_:
            assert not _passes_early(ct, np_, shape.accumulators(np_, cn)), (ct, cn, np_)
            fused += 1
    assert fused > 16 and shape.parts(512, 256) == 128 and shape.parts(384, 192) == 192 and shape.parts(320, 192) == 64
