"""Source rule of the kernels of the multigrid PCG loop, which start before their predecessor has ended (CPU; a race is
not provoked on a GPU).  Every operand that a kernel of the loop writes must be read after griddepcontrol.wait: a
parameter that is declared __restrict__ and only read counts as constant during the kernel, so its load may take the
read-only path and be moved across the wait.  Stencils and tables, which no kernel of the loop writes, are read with
__ldg or through local pointers.  And no CTA leaves before the wait: a kernel's reads before its own wait rest on every
CTA of its predecessor having waited."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pict_b200", "csrc", "multigrid.cu")


def _strip(text):
    return re.sub(r"//[^\n]*", "", text)


def _matched(text, i, opening, closing):
    depth = 0
    for k in range(i, len(text)):
        depth += (text[k] == opening) - (text[k] == closing)
        if depth == 0:
            return k
    raise ValueError("unbalanced")


def _kernels():
    """name -> (parameter list, body) of every __global__ function."""
    text = _strip(open(SRC).read())
    out = {}
    for m in re.finditer(r"__global__\s+void\b", text):
        k = text.index("k_", m.end())
        name = re.match(r"\w+", text[k:]).group(0)
        p0 = text.index("(", k)
        p1 = _matched(text, p0, "(", ")")
        b0 = text.index("{", p1)
        out[name] = (text[p0:p1 + 1], text[b0:_matched(text, b0, "{", "}") + 1])
    return text, out


def _loop_kernels():
    text, kernels = _kernels()
    names = set()
    for m in re.finditer(r"\bmg_launch\(", text):
        names |= set(re.findall(r"\bk_\w+", text[m.end() - 1:_matched(text, m.end() - 1, "(", ")")]))
    return {n: kernels[n] for n in names if n in kernels}


def test_loop_kernels_are_found():
    assert {"k_mg_restrict", "k_mg_prolong", "k_mg_restrict2", "k_mg_prolong2", "k_mg_subcycle", "k_pcg_spmv_dot",
            "k_pcg_spmv_dot_bulk", "k_pcg_dot4", "k_pcg_scalars", "k_pcg_update", "k_pcg_report",
            "k_pcg_loop_cond"} <= set(_loop_kernels())


@pytest.mark.parametrize("name", sorted(_loop_kernels()))
def test_no_operand_is_declared_read_only(name):
    params, _ = _loop_kernels()[name]
    assert "__restrict__" not in params


@pytest.mark.parametrize("name", sorted(_loop_kernels()))
def test_no_return_before_the_wait(name):
    _, body = _loop_kernels()[name]
    wait = re.search(r"\bmg_pdl_(?:entry|wait)\(\);", body)
    assert wait, "does not wait for its predecessor"
    assert not re.search(r"\breturn\b", body[:wait.start()])


def test_no_member_of_an_operand_struct_is_declared_read_only():
    text, _ = _kernels()
    for m in re.finditer(r"\bstruct\s+(\w+)\s*\{", text):
        body = text[m.end() - 1:_matched(text, m.end() - 1, "{", "}")]
        assert "__restrict__" not in body, m.group(1)
