"""Shared memory that a thread of one CTA of a pair writes for matrix instructions that the other CTA issues: the arrival that publishes it
releases at cluster scope and the wait for it acquires there.  Read from the source: a missing one need not show in any run."""

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "csrc"


def _body(text: str, name: str) -> str:
    start = re.search(rf"__forceinline__ \w+ {name}\(", text).start()
    return text[start : text.index("\n}\n", start)]


def test_cleared_rows_are_released_to_the_other_cta():
    common, kernel = (CSRC / "pair_common.cuh").read_text(), (CSRC / "grouped_wgrad_tcgen05_2cta.cu").read_text()
    kernel = re.sub(r"//[^\n]*", "", kernel)
    arrivals, waits = re.findall(r"(\w+)\(ready_bar\(s\), 0\)", kernel), re.findall(r"(\w+)\(ready_bar\(s\), \(", kernel)
    assert len(arrivals) == 1 and len(waits) == 1
    assert "mbarrier.arrive.release.cluster.shared::cluster" in _body(common, arrivals[0])
    assert "mbarrier.try_wait.parity.acquire.cluster" in _body(common, waits[0])
    cleared = kernel[: kernel.index(f"{arrivals[0]}(ready_bar")]
    assert cleared.rindex("fence_async_smem()") > cleared.rindex("st.shared.v4.b32")
