"""Kernels that wait for the kernel before them in the stream (kernel_begin /
kernel_wait) read memory that is written during their own lifetime: neither
they nor the device functions they call may mark it read-only or unaliased
(__ldg, __restrict__), since such loads may be moved ahead of the wait."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "autoquantizer_b200", "csrc")


def _source(name):
    text = open(os.path.join(CSRC, name)).read()
    text = re.sub(r"//[^\n]*", "", text)
    return re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "", text)


def _functions(text):
    """(name, signature and body) of every device function and kernel."""
    for m in re.finditer(r"\b__(?:global|device)__\b[^;{}]*?\b(\w+)\s*\([^;{}]*\)[^;{}]*\{", text):
        depth, k = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[k], 0)
            k += 1
        yield m.group(1), text[m.start():k]


@pytest.mark.parametrize("name,kernels", [
    ("aq_sim.cu", {"k_bin", "k_scatter", "k_items", "k_scan_sums", "k_scan_top", "k_scan_apply"}),
    ("aq_adjoint.cu", {"k_ad_pass", "k_ad_g2p_bwd", "k_ad_p2g_bwd"}),
    ("aq_kernels.cuh", {"k_step"}),
])
def test_no_read_only_loads_behind_a_wait(name, kernels):
    found = dict(_functions(_source(name)))
    waiting = {k for k, text in found.items() if re.search(r"\bkernel_(begin|wait)\s*\(\)", text)}
    waiting -= {"kernel_begin", "kernel_wait"}
    assert waiting == kernels
    # what they call, from this file and from the headers they share
    for h in ("aq_kernels.cuh", "aq_codec.cuh"):
        found.update(_functions(_source(h)))
    reached, todo = set(), set(waiting)
    while todo:
        f = todo.pop()
        reached.add(f)
        todo |= {g for g in re.findall(r"\b(\w+)\s*(?:<[^;(){}]*>)?\s*\(", found[f]) if g in found} - reached
    bad = {f for f in reached if "__ldg" in found[f] or "__restrict__" in found[f]}
    assert not bad, bad
