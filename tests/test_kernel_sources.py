"""Rules of the kernels that a run cannot show without failing on the GPU, read from the sources."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "lightly_trian_quant_b200" / "csrc"


def test_warps_wait_with_one_decision():
    """a wait that runs out must not divide a warp: lanes that leave and lanes that go on to a warp-wide instruction would wait for each other without
    a limit.  The wait of a single thread stays in the headers that build the others on it and in the peak probes, where one thread works alone."""
    alone = {"kf_sm100.cuh", "kf_sm100_pair.cuh", "kf_peak.cu"}
    single = [f"{path.name}:{no}: {line.strip()}" for path in sorted(CSRC.glob("*.cu*")) if path.name not in alone
              for no, line in enumerate(path.read_text().splitlines(), 1) if re.search(r"\bmbar_wait(_cluster)?\(", line.split("//")[0])]
    assert not single, single
