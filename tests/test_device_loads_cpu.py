"""How the kernels may read memory, checked on their sources.

Most kernels are launched programmatically: they are resident while the launch in front of them still runs, and wait
(pdl_wait) before they touch what it writes.  A non-coherent load (__ldg) is only defined for memory that nobody writes during the
kernel's lifetime, so it is left to constants: weights, their scales, biases, norms and rotation tables."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "zeninfer_b200", "csrc")
CONSTANTS = {"base", "bias", "w", "wsrc", "uw_row", "sw_row", "s32_row", "o32_row", "d_row", "cos_t", "sin_t", "dt_bias", "a_log", "decay", "norm"}


def _source(name):
    return re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())


@pytest.mark.parametrize("name", sorted(os.path.basename(f) for f in glob.glob(os.path.join(CSRC, "*.cu*"))))
def test_non_coherent_loads_are_of_constants(name):
    for what in re.findall(r"__ldg\(\s*(?:reinterpret_cast<[^>]*>\()?\s*([\w.>-]+)", _source(name)):
        assert re.split(r"\.|->", what)[-1] in CONSTANTS, f"{name}: __ldg of {what}"


# Arguments declared const and __restrict__ may become non-coherent loads by themselves: what the launch in front writes is then
# asked for with __ldcg.
@pytest.mark.parametrize("name,kernel,argument", [("gemm_groups.cuh", "group_digits_acts_kernel", "x"), ("attention_tc.cuh", "attention_prefill_tc_kernel", "q"),
                                                  ("attention_tc.cuh", "attention_prefill_tc_kernel", "pos_ptr")])
def test_what_the_launch_in_front_writes_is_read_coherently(name, kernel, argument):
    text = _source(name)
    body = text[text.index(kernel + "("):]
    body = body[body.index(") {"):]
    made = re.findall(rf"(\w+) = reinterpret_cast<const float4\*>\({argument} \+", body)      # pointers formed from it
    for start in [argument, *made]:
        assert not re.search(rf"\*{start}\b(?!\*)|\b{start}\[|\*reinterpret_cast<const float4\*>\({start}\b", body), f"{kernel}: plain load of {start}"
    assert re.search(rf"__ldcg\((?:reinterpret_cast<const float4\*>\()?(?:{'|'.join([argument, *made])})\b", body)


def test_a_decode_product_reads_only_weights_before_the_launch_in_front_has_ended():
    """Bias, norm weights, shift and output norm may be what the launch in front writes: up to the wait they are asked into L2 at most."""
    text = _source("gemv_bf16.cuh")
    body = text[text.index("gemv_bf16_kernel("):]
    before = body[:body.index("pdl_wait();")]
    assert not re.search(r"__ldg|__ldcg|row_words\(|sublayer_", before), "loads in front of the wait"
    for called in set(re.findall(r"\b(prologue_\w+)\(", before)):
        of = text[text.index(called + "("):]
        assert not re.search(r"__ldg|__ldcg|row_words\(", of[:of.index("\n}\n")]), f"{called}: loads in front of the wait"
