"""CPU: the Python setters' defaults are the library's, so that setting one value leaves the others as they were."""
import inspect
import os
import re

import voronoids_gb300 as V

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_schedule_defaults():
    src = open(os.path.join(ROOT, "voronoids_gb300", "csrc", "vd_capi.cu")).read()
    tree = src[src.index("struct vd_tree {"):]
    args = inspect.signature(V.DelaunayTree.set_schedule).parameters
    for name, p in args.items():
        if name != "self":
            assert float(re.search(rf"\b{name} = ([\d.]+);", tree).group(1)) == p.default, name
    header = open(os.path.join(ROOT, "include", "voronoids_gpu.h")).read()
    doc = re.search(r"Defaults ([\d.]+), ([\d.]+) and ([\d.]+)\. \*/\s*int vd_set_schedule", header).groups()
    assert [float(x) for x in doc] == [p.default for n, p in args.items() if n != "self"]
