"""Which kernel a bounded wait that ran out is reported for, from the sources: no GPU."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "pygpukit_b200" / "csrc"


def test_every_kernel_with_bounded_waits_is_reported_by_a_name_of_its_own():
    """A word per source file, a name per word: the call that synchronises names the entry point whose results are not valid."""
    kinds = re.search(r"enum WaitKind \{([^}]*)\}", (CSRC / "common.cuh").read_text(encoding="utf-8")).group(1)
    kinds = [k.strip() for k in kinds.split(",")][:-1]
    names = re.search(r"what\[kWaitKinds\] = \{([^}]*)\}", (CSRC / "runtime.cu").read_text(encoding="utf-8")).group(1)
    names = re.findall(r'"(\w+)"', names)
    assert len(names) == len(kinds) == len(set(names))
    users = {k: [f.name for f in sorted(CSRC.glob("*.cu")) if f"wait_word({k})" in f.read_text(encoding="utf-8")] for k in kinds}
    assert all(len(u) == 1 for u in users.values()), users
    assert dict(zip(kinds, names))["kWaitLinear"] == "seq_linear_attention_chunks" and users["kWaitLinear"] == ["seq_linear_tc.cu"]
    assert dict(zip(kinds, names))["kWaitPrompt"] == "sdpa_causal_fixed_cache" and users["kWaitPrompt"] == ["attention_tc.cu"]
    assert dict(zip(kinds, names))["kWaitFp8Rows"] == "gemm_fp8_rows" and users["kWaitFp8Rows"] == ["gemm_tc_rows.cu"]
