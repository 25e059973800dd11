"""Kernels launched as programmatic dependents touch the fields only after their wait for the
previous kernel: every __restrict__ pointer to a field, through which the compiler may move an
access above the wait, goes through pdl_enter."""
import glob
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "steamroller.jl_b200", "csrc")
# read-only tables, uploaded and waited for by the host
TABLES = {"coord_of", "src", "tw", "hw", "f", "lvs", "ent"}


def kernels():
    """name -> (pointer parameters, those that are __restrict__, body)."""
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*\)\s*)?(\w+)\s*\(", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(text[i], 0)
                i += 1
            params = text[m.end():i - 1]
            depth, j = 1, text.index("{", i) + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[j], 0)
                j += 1
            pointers = [p for p in params.split(",") if "*" in p]
            out[m.group(1)] = ([re.search(r"(\w+)\s*(?:=.*)?$", p.strip()).group(1) for p in pointers],
                               [re.search(r"(\w+)\s*(?:=.*)?$", p.strip()).group(1) for p in pointers if "__restrict__" in p],
                               text[i:j])
    return out


def test_fields_are_touched_after_the_wait():
    text = "".join(open(p).read() for p in glob.glob(os.path.join(CSRC, "*.cu*")))
    launched = set(re.findall(r"launch_pdl\(\s*(\w+)", text)) | {"k_gs_push", "k3_gs_push", "k3_interp_push"}
    seen = kernels()
    wrong = []
    for name in sorted(launched & set(seen)):
        pointers, restricted, body = seen[name]
        enter = re.search(r"pdl_enter\(([^)]*)\)", body)
        if enter:
            after = {a.strip() for a in enter.group(1).split(",")}
            missing = [p for p in pointers if p not in after | TABLES]
        elif "griddepcontrol.wait" in body:
            missing = [p for p in restricted if p not in TABLES]
        else:
            missing = ["no wait"]
        if missing:
            wrong.append((name, missing))
    assert len(launched & set(seen)) > 20 and not wrong, wrong
