"""tests/native/split_check.cu on the CPU: the integer split of FP64 values into
two and three FP32 values (meshoid_gb300/csrc/mg_split.cuh) equals the FP64
conversions and subtractions bit for bit, at every exponent."""
from test_native_helpers import _build_and_run


def test_split_equals_fp64_conversions(tmp_path):
    _build_and_run(tmp_path, "split_check")
