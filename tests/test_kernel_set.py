"""The library compiles the transform kernels that a plan can launch and no others: the first
kernel of a process loads the whole module, so each unused one makes the first handle slower."""

import re
import subprocess

import pytest

from materialite_b200 import _native as nat

# kernel: index of the argument that selects the projection (PRO_* forward, EPI_* inverse)
PASSES = ["zfwd_kernel", "zinv_kernel", "zyfwd_kernel", "yzinv_kernel", "zyfwd_cl_kernel",
          "yzinv_cl_kernel"]
# (transform, storage): projections. Given field 0/0, residual 1/1, re-projection 4/3, Krylov 5/4
FORWARD = {("double", "double"): {0, 1, 5}, ("float", "float"): {0, 5}, ("double", "float"): {1, 4}}
INVERSE = {("double", "double"): {0, 1, 4}, ("float", "float"): {0, 4}, ("double", "float"): {1, 3}}


def kernels():
    try:
        out = subprocess.run(["nm", "-C", nat.library_path()], check=True, capture_output=True,
                             text=True).stdout
    except FileNotFoundError:
        pytest.skip("no nm")
    return {(m[1], m[2]) for m in re.finditer(r"void (\w+_kernel)<([^>]*)>\(", out.replace("(int)", "").replace("(bool)", ""))}


def test_transform_kernels_are_those_of_the_projections():
    seen = kernels()
    assert seen
    for name, args in seen:
        a = [x.strip() for x in args.split(",")]
        if name in PASSES:
            allowed = (FORWARD if "fwd" in name else INVERSE)[a[0], a[1]]
            assert int(a[2]) in allowed, (name, args)
        if name in ("xpass_kernel", "ypass_kernel") and a[0] != a[1]:
            # Krylov iterations run in the storage type
            assert a[3 if name == "ypass_kernel" else 2] in ("0", "false"), (name, args)
