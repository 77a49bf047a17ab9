"""The kernel launches that bench.py reports per force call, against the
launches in the library's sources: the kernels named in each form's launch
function, the zeroing before them where force_calc does it, and the reduction
of the totals behind them."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _read(*p):
    return re.sub(r"//[^\n]*", "", open(os.path.join(ROOT, *p)).read())


def _body(text, name):
    k = text.index(name + "(")
    k = text.index("{", text.index(")", k))
    depth, e = 0, k
    while True:
        depth += {"{": 1, "}": -1}.get(text[e], 0)
        e += 1
        if depth == 0:
            return text[k:e]


def _kernels(body):
    return set(re.findall(r"launch_(?:dep|full)\((k\w+)", body)) | set(re.findall(r"(k_\w+)<[^;<]*><<<", body))


def test_launches_per_force_call():
    csrc = ("mapp_b200", "csrc")
    said = re.search(r'"gpu_launches": \{"fp64": (\d+), "fp32": (\d+), "mlp": (\d+)\}', open(os.path.join(ROOT, "bench.py")).read())
    said = [int(v) for v in said.groups()]
    call = _body(_read(*csrc, "mg_api.cu"), "int mg_ff_force_calc")
    assert call.count("launch_reduce_partials(") == 1 and "if (!f32) CU(launch_zero(" in call
    fp64 = _kernels(_body(_read(*csrc, "mg_dmd.cu"), "cudaError_t dmd_force_nt"))
    d32 = _read(*csrc, "mg_dmd32.cu")
    fp32, tail = _kernels(_body(d32, "cudaError_t dmd32_force_nt")), _kernels(_body(d32, "cudaError_t dmd32_tail_nt"))
    mlp = _kernels(_body(_read(*csrc, "mg_mlp_tc.cu"), "cudaError_t mlp_force_nt"))
    assert said == [1 + len(fp64) + 1, len(fp32) + 1, 1 + len(mlp) + len(tail) + 1]
