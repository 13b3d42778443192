"""tests/kernel_args.py: the sources' parameter lists, and names as the compiler forms them."""
import pytest

from tests.kernel_args import arguments, parameters


def test_parameters():
    assert parameters("mi8_gemm_pair_kernel") == ["kP8", "kMaps", "kResident", "kHalves"]
    names = parameters("mi8_gemm_kernel")
    assert names[0] == "TM" and "kBelow" in names and len(set(names)) == len(names)


def test_arguments():
    mangled = "_ZN3mi883_GLOBAL__N__0020mi8_gemm_pair_kernelILb0ELi1ELb0ELb1EEEvv"
    assert arguments("mi8_gemm_pair_kernel", mangled) == {"kP8": 0, "kMaps": 1, "kResident": 0, "kHalves": 1}
    assert arguments("mi8_gemm_kernel", mangled) is None
    with pytest.raises(AssertionError):
        arguments("mi8_gemm_pair_kernel", mangled.replace("Lb1EE", "E"))
