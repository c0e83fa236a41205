"""Kernels that start with chain_wait() may be resident while an earlier kernel
of their chain still writes, so they must not declare as read-only what the chain
writes: __ldg and const __restrict__ only for the systems' tables."""
import os
import re

import pytest

from conftest import PKG

STATIC = {"sid", "sys", "row"}  # written before the chain starts, by kernels it waits for


def _kernels():
    src = open(os.path.join(PKG, "csrc", "nd_md.cu")).read()
    out = {}
    for m in re.finditer(r"^__global__", src, re.M):
        k = src.index("{\n", m.end()) + 2
        head, body, depth = src[m.start():k], k, 1
        while depth:
            depth += {"{": 1, "}": -1}.get(src[k], 0)
            k += 1
        text = src[body:k]
        if "chain_wait();" in text:
            out[re.search(r"(k_\w+)\(", head).group(1)] = (head, text)
    return out


KERNELS = _kernels()


def test_chained_kernels_found():
    assert {"k_md_place", "k_md_block_union", "k_md_block_lists", "k_md_leaf_lists",
            "k_md_step"} <= set(KERNELS)


@pytest.mark.parametrize("name", sorted(KERNELS))
def test_no_read_only_loads_of_what_the_chain_writes(name):
    head, body = KERNELS[name]
    for text in (head, body):
        loads = re.findall(r"__ldg\(\s*[&*]?(?:a\.)?(\w+)", text)
        assert set(loads) <= STATIC, set(loads) - STATIC
        const = re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", text)
        assert set(const) <= STATIC, set(const) - STATIC


def test_steps_read_only_loads_follow_the_chaining():
    # the step kernel's loads go through step_ld, read-only where the step does not
    # wait inside the chain; the host chains exactly those that do
    src = open(os.path.join(PKG, "csrc", "nd_md.cu")).read()
    head, body = KERNELS["k_md_step"]
    assert "constexpr bool CHAIN = kStepChained<TPA>;" in body
    assert "if constexpr (MODE == 0 && CHAIN) chain_wait();" in body
    assert set(re.findall(r"step_ld<(\w+)>", body)) == {"CHAIN"}
    assert "constexpr bool kStepChained = TPA > 1;" in src
    assert "chained = MODE == 0 && m->gated && m->nsys == 0 && m->tpa > 1;" in src


def test_step_arguments():
    text = open(os.path.join(PKG, "csrc", "nd_md_engine.cuh")).read()
    args = text[text.index("struct StepArgs"):text.index("struct MDEngine")]
    const = set(re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", args))
    assert const <= STATIC | {"im"}, const
