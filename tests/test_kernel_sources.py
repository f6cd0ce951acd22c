"""Orderings between kernels and blocks that no run can show to be missing, held in the kernel sources themselves."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "qw38_b200" / "csrc"


def code(path):
    """The source without its comments."""
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", path.read_text(), flags=re.S)


def test_minima_are_published_across_the_cluster():
    """mmq_f16.cu: ordinary stores of both blocks that the leader's MMA reads.  Proxy fence, release and arrival on the writers'
    side, acquire between the wait for the same stage and the MMA on the issuer's."""
    text = code(CSRC / "mmq_f16.cu")
    writer = text[text.index("sts128(smem + C::oMins"):]
    assert writer.index("fence.proxy.async") < writer.index("release_shared();") < writer.index("arrive_cluster(a_full0")
    issuer = text[text.index("mbar_wait_inline_relaxed_cluster(a_full"):]
    assert issuer.index("acquire_shared();") < issuer.index("mma_pair_ss(")
