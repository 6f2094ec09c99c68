"""The bench names and rates the kernel that ran, not the one its tuning suggests."""
import importlib.util
import os

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("bench", os.path.join(ROOT, "bench.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


# the FP64 form with an empty tuning takes the FP64 instructions where data or
# free memory rule the tensor cores out
@pytest.mark.parametrize("form,kernels,name,products", [
    ("fp64", ["tensor_core"], "triples_tc_kernel", 36),
    ("fp64", ["fp64_instructions"], "triples_fp64_kernel", 1),
    ("fp64", ["fp64_instructions"] * 4 + ["tensor_core"] * 92, "triples_tc_kernel", 36),
    ("fp64", ["fp64_instructions"] * 3 + ["tensor_core"], "triples_fp64_kernel", 1),
    ("split_f16", ["split"], "triples_split_kernel", 3),
    ("split_f16", ["tensor_core"], "triples_tc_kernel", 3)])
def test_roofline_of_the_kernel_that_ran(bench, form, kernels, name, products):
    peaks = {"bf16_tflops": 1900.0}
    kernel = bench._kernel_name(form, kernels)
    r = bench._roofline(form, 2, 1e12, 1000.0, peaks, 1.25, None, kernel)
    assert r["kernel"] == kernel == name
    assert r["achieved"] == pytest.approx(products)
    assert r["peak"] == (1.25 if products == 1 else 1900.0)
