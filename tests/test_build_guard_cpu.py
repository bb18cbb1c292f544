"""The build refuses register spills in the kernels that keep tensor-memory loads in flight, and in no others."""

import re

import pytest

from oops_b200.csrc.build import CSRC, NO_SPILL_KERNELS, _spilling_entries

# names as nvcc mangles them: kernels live in anonymous namespaces, which carry their file's name
ENTRIES = {
    "fused": "_ZN7oops_ta55_GLOBAL__N__87b3404d_22_ta_tensor_bwd_sm100_cu_2e2a600819ta_bwd_fused_kernelI6__halfLb1ELb0ELb1EEEvNS0_7FParamsE",
    "forward": "_ZN7oops_ta51_GLOBAL__N__af6a735c_18_ta_tensor_sm100_cu_b47f75aa13ta_fwd_kernelI6__halfLb1ELb0ELb1ELb0EEEvNS0_9FwdParamsE",
    "bias": "_ZN7oops_ta55_GLOBAL__N__87b3404d_22_ta_tensor_bwd_sm100_cu_2e2a600819ta_bwd_dbias_kernelI6__halfLi2EEEvNS0_8DbParamsE",
    "norm": "_ZN7oops_ta49_GLOBAL__N__a00203c3_16_ta_layer_norm_cu_307876c430layer_norm_forward_rows_kernelI13__nv_bfloat16S2_Li8ELi1ELi16EEEvv",
}


def log(spilling):
    """What ptxas says about the entries, `spilling` of which store 44 bytes."""
    lines = []
    for key, name in ENTRIES.items():
        count = 44 if key in spilling else 0
        lines += [f"ptxas info    : Compiling entry function '{name}' for 'sm_100a'", f"ptxas info    : Function properties for {name}",
                  f"    48 bytes stack frame, {count} bytes spill stores, {count} bytes spill loads", "ptxas info    : Used 96 registers"]
    return "\n".join(lines)


@pytest.mark.parametrize("key", ["fused", "forward", "bias"])
def test_a_guarded_kernel_that_spills_is_named(key):
    found = _spilling_entries(log({key, "norm"}), NO_SPILL_KERNELS)
    assert len(found) == 1 and ENTRIES[key] in found[0] and "44 bytes" in found[0]


def test_no_others_are():
    assert _spilling_entries(log({"norm"}), NO_SPILL_KERNELS) == []
    assert _spilling_entries(log(set()), NO_SPILL_KERNELS) == []


def test_the_guarded_names_are_those_of_the_sources():
    sources = "".join(path.read_text() for path in CSRC.glob("*.cu"))
    for name in NO_SPILL_KERNELS:
        assert re.search(rf"__global__[^;{{]*\b{name}\(", sources), name
