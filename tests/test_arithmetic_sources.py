"""The FP16-storage path keeps its arithmetic in FP32 as written: which kernels
may use the approximate division and root instructions."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "glasscamerapublic_b200" / "csrc"
APPROX = r"__fdividef|__frcp|__frsqrt|\brsqrtf\(|\b(?:sqrt|rsqrt|rcp|div)\.approx"


def code(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


def test_the_raw_front_end_divides_and_takes_roots_in_full_precision():
    assert re.findall(APPROX, code("gls_front.cu")) == []


def test_the_block_matchers_constants_are_formed_in_full_precision():
    """Of the approximate forms only 1 / sqrt(2 log2 e), a constant of the weights' scale."""
    found = re.findall(r"[^\n]*(?:" + APPROX + r")[^\n]*", code("gls_blockmatch.cu"))
    assert found and all("isq = rsqrtf(lk);" in line for line in found)
