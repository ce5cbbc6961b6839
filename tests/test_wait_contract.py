"""The no-hang contract of the prefill kernels, read from their source (a completion that never comes is
nothing a test can stage without hanging a kernel): a wait without a clock of its own ends only when another role raises the abort flag, so
behind each completion that such a wait depends on some role must wait with a clock."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flash_attention_b200", "csrc")


def _role(name, banner):
    """The code of one role, from its banner to the next one, without comments."""
    text = open(os.path.join(CSRC, name)).read()
    parts = re.split(r"// =+ (.+?) =+\n", text)
    roles = {parts[i].strip(): parts[i + 1] for i in range(1, len(parts) - 1, 2)}
    return re.sub(r"//.*", "", roles[banner])


@pytest.mark.parametrize("name,banner", [("attn_ws64.cuh", "TMA loaders"), ("attn_ws.cuh", "PV issuer")])
def test_the_last_product_of_a_cta_is_awaited_with_a_clock(name, banner):
    """The last P V of a CTA's last tile: its reader waits by the flag alone, and no issuer has anything
    behind it to wait for.  One of the roles with a clock waits for it, after its tile loop and before its drain."""
    loop, drain = _role(name, banner).split("ti += 1;")
    tail = drain[:drain.index("kDrain")]
    assert re.search(r"\bmbar_wait(_relaxed<\w+>)?\(bars\.at\(Bars::kPvDone", tail), "no bounded wait behind the last product"
    assert "mbar_wait_flag" not in loop + drain


@pytest.mark.parametrize("name", ["attn_decode.cuh", "aux_kernels.cuh", "quantize.cuh"])
def test_the_other_kernels_wait_with_a_clock_only(name):
    assert "mbar_wait_flag" not in open(os.path.join(CSRC, name)).read()


def test_a_decode_warp_writes_only_its_own_hand_over_slot():
    """Slot (wg, wq) is read by warp wq of the other warpgroup, and only its own hand-over barrier orders that
    reader before the next write: a write by any other warp could come before the read."""
    text = re.sub(r"//.*", "", open(os.path.join(CSRC, "attn_decode.cuh")).read())
    writes = re.findall(r"if \(([^\n]*?)\) s_hand\[([^\n]+?)\] = ", text)
    assert len(writes) == text.count("s_hand[") - len(re.findall(r"= s_hand\[", text)) == 2
    k_max_rows, k_r = 32, 8
    for cond, index in writes:
        for wg in (0, 1):
            for wq in range(4):
                for lane in range(k_r):
                    env = {"wg": wg, "wq": wq, "lane": lane, "my_row": lane, "kR": k_r, "kMaxRows": k_max_rows}
                    if eval(cond.replace("&&", "and"), env):
                        assert eval(index, env) == (wg * 4 + wq) * k_max_rows + lane, (cond, index, wg, wq)
