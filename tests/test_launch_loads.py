"""Kernels queued with an overlapping start (launch_dep, launch_full, or the
launch attribute itself) are resident while the kernel before them still
writes: by the sources, none of them takes a const __restrict__ pointer (which
the compiler may read through the read-only path), the explicit read-only
loads are those of the potential tables, and the wait comes first."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mapp_b200", "csrc")
SRC = {os.path.basename(p): open(p).read() for p in sorted(glob.glob(os.path.join(CSRC, "*.cu*")))}
# kernels launched through a function pointer (kA, kB, kf)
BY_POINTER = {"k_dmd32_dens", "k_dmd32_force", "k_dmd32_fill"}
# reads nothing that a queued kernel writes before its wait (comments at the kernels)
WAITS_LATER = {"k_mlp_train", "k_mlp_adam"}


def _strip(text):
    return re.sub(r"//[^\n]*", "", text)


def _queued():
    out = set(BY_POINTER)
    for text in SRC.values():
        t = _strip(text)
        out |= set(re.findall(r"launch_(?:dep|full)\(\s*(k_\w+)", t))
        out |= set(re.findall(r"cudaLaunchKernelEx\(&cfg,\s*(k_\w+)", t))
    return out


def _kernels():
    """name -> (parameter list, first statement) of every __global__ definition."""
    out = {}
    for text in SRC.values():
        t = _strip(text)
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*\)\s*|MG_\w+\s+)?(k_\w+)\s*\(", t):
            depth, k = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(t[k], 0)
                k += 1
            body = t[k:].lstrip()
            if body.startswith("{"):
                out[m.group(1)] = (t[m.end():k - 1], body[1:].lstrip().split(";")[0].strip())
    return out


def test_every_queued_kernel_is_found():
    missing = _queued() - set(_kernels())
    assert not missing and len(_queued()) > 40


@pytest.mark.parametrize("name", sorted(_queued()))
def test_parameters_and_wait(name):
    params, first = _kernels()[name]
    for p in params.split(","):
        assert not ("const" in p.split("*")[0] and "__restrict__" in p), p.strip()
    if name not in WAITS_LATER:
        assert first == "dep_sync()"


def test_read_only_loads_are_the_tables():
    found = set()
    for name, text in SRC.items():
        for ln in _strip(text).splitlines():
            if "__ldg(" in ln or "ld.global.nc" in ln:
                found.add((name, re.sub(r"\s+", " ", ln.strip())))
    for name, ln in found:
        table = "d.pkS" in ln or (name == "mg_dmd_common.cuh" and ("return __ldg(p);" in ln or '"l"(row)' in ln))
        assert table, (name, ln)


def test_the_audit_starts_after_the_network():
    """Blocks of the learned form's audit that wait beside the persistent network
    kernel slow it down (1 % of a 500000-site call): a plain launch."""
    assert "k_mlp_audit" not in _queued()
    assert "k_mlp_audit<NT, 3><<<" in SRC["mg_mlp_tc.cu"]


def test_the_first_training_step_is_a_plain_launch():
    """k_mlp_train reads its rows before its wait, so the step that follows the
    kernels filling them must not be queued early."""
    t = _strip(SRC["mg_mlp.cu"])
    body = t[t.index("cudaError_t launch_mlp_train_step("):]
    first = body[body.index("if (step == 0 || fixed) {"):]
    first = first[:first.index("}")]
    assert "k_mlp_train<<<" in first and "launch_dep" not in first
    assert body.index("launch_dep(k_mlp_train") > body.index("} else")
    api = _strip(SRC["mg_api.cu"])
    grad = api[api.index("int mg_mlp_grad("):]
    grad = grad[:grad.index("launch_mlp_train_step(")]
    assert grad.count("cudaMemcpyAsync(") == 2 and "cudaMemcpy(" not in grad  # on the step's own stream
