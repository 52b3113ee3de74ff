"""What can be seen of the kernels without a GPU: rules that their source files keep."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "garlic_inference_b200" / "csrc"
SPINNING = sorted(p.name for p in CSRC.glob("*.cu") if "_SPIN_LIMIT" in p.read_text())


def _bodies(text):
    """(name, body) of every __global__ function."""
    for m in re.finditer(r"__global__[^;{]*?(\w+)\s*\([^{;]*\)\s*\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), text[m.end():i - 1]


@pytest.mark.parametrize("name", SPINNING)
def test_no_barrier_without_a_limit_between_bounded_waits(name):
    """A warp that gives up a bounded wait leaves its role for the block's last barrier.  A barrier of the hardware's between the
    waits would hold the warps that did not give up for good: warps may meet there only before the first wait."""
    found = False
    for kernel, body in _bodies((CSRC / name).read_text()):
        waits = [m.start() for m in re.finditer(r"mbar_wait\(|wait_warp\(", body)]
        if not waits:
            continue
        found = True
        between = re.sub(r"//[^\n]*", "", body[waits[0]:waits[-1]])
        assert not re.search(r"\bbar\.(cta\.)?(sync|red)|\bbarrier\.(cta\.)?(sync|red)|__syncthreads|__syncthreads_", between), kernel
    assert found, f"{name}: no kernel with bounded waits was recognised"


def test_every_code_of_a_kernel_that_gave_up_is_explained(monkeypatch):
    """The message names each code that the sources can put into the error flag, alone or in a range."""
    import torch
    from garlic_inference_b200.ops import kernels
    codes = {int(c) for p in CSRC.glob("*.cu") for c in re.findall(r"#define \w+_ERR_\w+ (\d+)", p.read_text())}
    assert len(codes) > 15
    flag = torch.zeros(1, dtype=torch.int32)
    monkeypatch.setattr(kernels, "tcgen05_error_flag", lambda device: flag)
    for code in sorted(codes):
        flag[0] = code
        with pytest.raises(kernels.WaitRanOut) as e:
            kernels.check_bounded_waits("cpu")
        said = str(e.value).split(":", 1)[1]
        ranges = [(int(a), int(b or a)) for a, b in re.findall(r"(?:^|, | )(\d\d)(?:-(\d\d))? [a-z]", said)]
        assert any(a <= code <= b for a, b in ranges), (code, ranges)
        assert int(flag) == 0
