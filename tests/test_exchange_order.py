"""The order of an exchange between resident tiles (os_tile.cuh, exchange): its
buffer in shared memory holds the band on the way out and then the ring on the
way in, in places that overlap, and warps run ahead of one another in the sweeps
between two exchanges. So each of the four steps has the CTA's barrier between
it and the next, and between the last one and the next exchange's first."""
import re

from tests.conftest import ROOT

SOURCE = ROOT / "opensayal_gb300" / "csrc" / "os_tile.cuh"


def exchange_body():
    text = SOURCE.read_text()
    at = text.index("__device__ __forceinline__ void exchange(")
    body = text[at:text.index("\n}\n", at)]
    return re.sub(r"//[^\n]*", "", body)


def test_a_barrier_lies_between_any_two_uses_of_the_buffer():
    uses = {"band in": r"exchange_patch<FIELDS, true, R>", "band out": r"packet_out\(true, p, ",
            "ring in": r"c\[0\] = make_float4\(", "ring out": r"exchange_patch<FIELDS, false, R>"}
    body = exchange_body()
    events = [(m.start(), "barrier") for m in re.finditer(r"__syncthreads\(\);", body)]
    for name, pattern in uses.items():
        found = [m.start() for m in re.finditer(pattern, body)]
        assert len(found) == 1, name
        events.append((found[0], name))
    order = [name for _, name in sorted(events)]
    assert order == ["barrier", "band in", "barrier", "band out", "barrier", "ring in", "barrier",
                     "ring out"]
