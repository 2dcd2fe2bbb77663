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


def test_a_pair_stays_until_its_commits_have_arrived():
    """the leader's commits release a stage in both CTAs, those of the last stages too, which nothing else waits for: the producer of each CTA goes once more
    round its ring of empty barriers before the cluster barrier behind which a CTA may leave."""
    text = (CSRC / "kf_gemm_pair.cu").read_text()
    producer = text[text.index("TMA producer (each CTA its own part)"):text.index("MMA issuer (leader)")]
    behind_the_loads = producer.rsplit("tma_load_2d_pair", 1)[1]
    assert "tc_commit_both(&empty[s])" in text
    assert re.search(r"for \(int i = 0; i < STAGES && ok; \+\+i\) \{\s*ok = mbar_wait_warp\(&empty\[s\], ph \^ 1, ", behind_the_loads), "no round of waits behind the last load"
