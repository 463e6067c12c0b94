"""Kernels whose blocks are placed while the launch before still runs
(griddepcontrol.wait): what that launch writes is not read-only for the whole of
such a kernel's life, so it may not be read through the read-only path (__ldg,
const __restrict__). Neither may a kernel so read what it writes itself. Checked
on the source of everything such a kernel calls."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dompap_gb300", "csrc")
# tables that no step and no training step writes: parameters of the masses and of
# the pairs, particle types and ids (the slots keep their order between rebuilds)
CONSTANT = ("a.mcoef", "a.mcoef_f", "a.sig_tab", "a.eps_tab", "a.isig_tab", "a.f32_tab", "a.types", "a.order", "tri")


def _source(name):
    with open(os.path.join(CSRC, name)) as fh:
        return re.sub(r"//[^\n]*", "", fh.read())


def _functions(text):
    """name -> its definitions (template heads included)."""
    out = {}
    for m in re.finditer(r"\b(\w+)\([^;{}()]*(?:\([^()]*\)[^;{}()]*)*\)\s*(?:const\s*)?\{", text):
        if m.group(1) in ("if", "for", "while", "switch"):
            continue
        depth, end = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        out.setdefault(m.group(1), []).append(text[m.start():end])
    return out


def _reached(functions, name):
    seen, todo = {}, [name]
    while todo:
        f = todo.pop()
        if f in seen or f not in functions:
            continue
        seen[f] = "\n".join(functions[f])
        todo += re.findall(r"\b(\w+)\s*(?:<[^;(){}]*>)?\(", seen[f])
    return seen


@pytest.mark.parametrize("files,kernels", [
    (("dp_common.cuh", "dp_integrate.cuh", "pair_kernels.cuh"), {"dp_step_lists"}),
    (("dp_common.cuh", "mlp_common.cuh", "mlp_train.cuh"), {"k_mlp_grad", "k_mlp_update"})])
def test_no_read_only_loads_of_live_data(files, kernels):
    functions = _functions("\n".join(_source(f) for f in files))
    waiting = {f for f, bodies in functions.items() for b in bodies
               if "griddepcontrol.wait" in b or re.search(r"\bdp_grid_wait\(\)", b)} - {"dp_grid_wait"}
    assert waiting == kernels
    for kernel in kernels:
        reached = _reached(functions, kernel)
        assert len(reached) > 1
        for name, body in reached.items():
            if name == "dp_fetch":  # plain when LIVE
                assert re.search(r"return LIVE \? \*p : __ldg\(p\);", body)
                continue
            assert "__restrict__" not in body, (kernel, name)
            for arg in re.findall(r"__ldg\(\s*([\w.]+)", body):
                assert arg in CONSTANT, (kernel, name, arg)
    if "dp_step_lists" in kernels:
        # and the overlapped kernel asks for plain loads all the way down
        assert "dp_step_split<32, false, true>" in "\n".join(functions["dp_step_lists"])
        split = "\n".join(functions["dp_step_split"])
        assert "dp_particle_sum<DP_ACC_FORCE, LANES, ALL, LIVE>" in split
        assert "dp_fetch<LIVE>(sh" in "\n".join(functions["dp_particle_sum"])
        assert "dp_fetch<true>(sh" in "\n".join(functions["dp_build_row"])


def test_replica_lists_are_read_with_plain_loads():
    """dp_batch_steps builds its lists and walks them in one launch."""
    body = "\n".join(_functions(_source("batch_kernels.cuh"))["dp_batch_steps"])
    assert "__ldg" not in body and "__restrict__" not in body
