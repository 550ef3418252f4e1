"""bench.py's clock samples cover a timed region shorter than nvidia-smi's start-up, and only that
region (a stand-in nvidia-smi on PATH; no GPU)."""

import os
import sys
import time

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FAKE = """#!{python}
import datetime, os, signal, sys, time
path = sys.argv[sys.argv.index("-f") + 1]
query = next(a for a in sys.argv if a.startswith("--query-gpu=")).split("=", 1)[1].split(",")
period = float(sys.argv[sys.argv.index("-lms") + 1]) / 1e3
rows = []
def done(*_):  # the rows reach the file when it ends
    open(path, "w").write("".join(rows))
    os._exit(0)
signal.signal(signal.SIGTERM, done)
time.sleep(0.3)
while True:
    mhz = "1965 MHz" if os.path.exists({marker!r}) else "315 MHz"
    now = datetime.datetime.now().strftime("%Y/%m/%d %H:%M:%S.%f")[:-3]
    known = {{"index": "0", "clocks.sm": mhz, "clocks.max.sm": "1965 MHz", "power.draw": "500 W", "timestamp": now}}
    rows.append(", ".join(known.get(q, "Not Active") for q in query) + "\\n")
    time.sleep(period)
"""


def test_a_short_region_is_sampled(tmp_path, monkeypatch):
    sys.path.insert(0, ROOT)
    import bench

    marker, fake = str(tmp_path / "running"), tmp_path / "nvidia-smi"
    fake.write_text(FAKE.format(python=sys.executable, marker=marker))
    fake.chmod(0o755)
    monkeypatch.setenv("PATH", f"{tmp_path}{os.pathsep}{os.environ['PATH']}")
    sampler = bench.ClockSampler(0)
    with sampler as clocks:
        time.sleep(0.05)  # the warm-up
        if hasattr(clocks, "mark"):
            clocks.mark()
        open(marker, "w").close()
        time.sleep(0.1)  # the timed region
    got = sampler.summary()
    assert got.get("samples", 0) >= 2, got
    assert got["sm_mhz"] == 1965.0 and got["reasons"] == [], got
