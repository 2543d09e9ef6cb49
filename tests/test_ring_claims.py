"""When a job ring runs down: by the host's late view of the claim cursor, which refused claims push past the
units there are and an admission puts back.  New work must never be taken for claimed work."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "cortexraytracercuda_b200" / "csrc"

MAIN = r"""
#include "rtc_claims.h"
#include <cstdio>
#define CHECK(x) if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; }
int main() {
    const uint32_t slots = 1000;
    rtc::RingClaims c;
    c.limit += 1500;                 // a job of 1,500 units, batch 0
    c.polled(0);
    CHECK(!c.runs_down(slots));      // nothing observed yet: all unclaimed
    c.polled(1);                     // batch 1
    c.observe(0, 1200, 1000);        // batch 0: 1,200 claimed
    CHECK(!c.runs_down(slots));      // 300 wait for slots
    c.polled(0);
    c.observe(1, 1780, 900);         // batch 1: all claimed, 280 claims refused
    CHECK(c.runs_down(slots));
    c.limit += 250;                  // a job of 250 units: every claim of it is still to come
    CHECK(!c.runs_down(slots));      // 900 live + 250 unclaimed
    c.polled(1);
    c.observe(0, 1790, 800);         // polled before the admission: the cursor says nothing of the new units
    CHECK(!c.runs_down(slots));      // 800 live + 250
    c.polled(0);
    c.observe(1, 1700, 1000);        // polled after it: the cursor was put back to 1,500
    CHECK(!c.runs_down(slots));      // 50 wait
    c.polled(1);
    c.observe(0, 1760, 900);
    CHECK(c.runs_down(slots));
    return 0;
}
"""


def test_runs_down_never_early(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "claims"
    subprocess.run([gxx, "-std=c++17", "-I", str(CSRC), str(tmp_path / "main.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
