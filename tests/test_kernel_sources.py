"""What the kernels' sources may not say, whatever they compute."""

import re
from pathlib import Path

KERNELS = Path(__file__).resolve().parent.parent / "fast_ulysses_b200" / "csrc" / "kernels"


def _sources():
    for path in sorted(KERNELS.iterdir()):
        if path.suffix in (".cu", ".cuh", ".h"):
            yield path.name, re.sub(r"//[^\n]*", "", path.read_text())


def test_kernels_that_overlap_their_predecessor_use_no_read_only_loads():
    """A kernel launched with launch_behind exists while the one before it still writes: loads that state the memory to be
    read-only for the kernel's lifetime are wrong there, and __ldg and __restrict__ also let the compiler move the load to before the
    wait. The one place left is the many-rank exchange's first move, in a kernel that is launched in the ordinary way."""
    found = {name: re.findall(r"ld\.global\.nc|ld_nc_v4|__ldg|__restrict__", text) for name, text in _sources()}
    assert found.pop("ptx.cuh") == ["ld_nc_v4", "ld.global.nc"]  # the helper itself
    assert found.pop("a2a4d.cu") == ["ld_nc_v4"]
    assert not any(found.values()), found
    a2a = dict(_sources())["a2a4d.cu"]
    assert "kCoherent ? ld_v4(from) : ld_nc_v4(from)" in a2a
    users = re.findall(r"ldst_move<false>", a2a)
    assert users and "launch_behind(a2a4d_kernel" not in a2a and a2a.count("a2a4d_kernel<false><<<") == 1
