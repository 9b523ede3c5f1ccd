"""Kernels that are started before the one ahead of them has ended may read through the
read-only path (__ldg) only what no kernel of the solve writes: the operator and its
sliced-ELL copy."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CONSTANT = re.compile(r"^(P\.(rowptr|col|val|sl_ptr|sl_row|sl_col|sl_val)|cp|vp)\b")


def test_read_only_loads_of_constant_data():
    src = open(os.path.join(ROOT, "usbs_gb300", "csrc", "lanczos.cu")).read()
    start = src.index("void st_pdl_prologue()")
    end = src.index("// per-CTA shared-memory layout of the cluster kernel")
    body = src[start:end]
    assert body.count("st_pdl_prologue();") >= 10
    args = re.findall(r"__ldg\(([^()]*)", body)
    assert args and all(CONSTANT.match(a.strip()) for a in args), args
    mode = src[src.index("int st_mode(const StreamCtl"):start]
    assert "__ldg(" not in mode
    # the two short names are pointers into the operator's copy
    assert re.search(r"const int\* cp = P\.sl_col", body)
    assert re.search(r"const VT\* vp = P\.sl_val", body)
