"""Kernels launched as programmatic dependents are alive while the kernel ahead of
them still writes.  What that one may write has to be read by plain loads through
pointers that are not __restrict__: __ldg, and const __restrict__ parameters, which
become read-only loads too, are for data that nothing writes during the kernel.

This reads the CUDA sources: every kernel that waits for the launch ahead (itself, or
in a function it calls) has no const __restrict__ parameter but the ones below, which
were complete before the launch ahead began, and uses __ldg on no others."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "fluid-sim_gb300" / "csrc"

# tables set by the host, and fields written two or more launches before (k_advect_sl_t
# and k_advect_sl_class are launched normally, after all that is ahead)
COMPLETE = {
    "k_advect_sl_t": {"u", "v"},
    "k_forcing": {"modes", "st"},
    "k_band_columns": {"lattice", "ex_u", "ex_v", "st"},
    "k_band_apply": {"ey_u", "ey_v"},
    "k_conv3x3": {"wpk", "bias"},
    "k_mg_up": {"rhs", "xin"},
    "k_loss_seed": {"out", "tgt"},
}
# device functions that read by __ldg where they are told that a field is complete, and
# who tells them so: the advected velocity, the up kernels' iterate and rhs
GUARDED = re.compile(r"COMPLETE \? __ldg")
TOLD = {
    "k_advect_sl_t": {"stage_tiles<2, true>", "TileView<true>"},
    "k_advect_sl_class": {"stage_tiles<2, true>", "TileView<true>"},
    "k_mc_combine_t": {"TileView<true>"},
    "k_mc_combine_class": {"TileView<true>"},
    "mg_up_reg": {"load<true>"},
    "trace_t": {"TileView<true>"},
    "trace_face": {"TileView<true>"},
    "advect_rows": {"TileView<true>"},
    "combine_rows": {"TileView<true>"},
}
WAIT = re.compile(r"pdl_wait\(\)|griddepcontrol\.wait")


def _block(s, i):
    """End of the braces that open at s[i]."""
    depth = 0
    for k in range(i, len(s)):
        depth += (s[k] == "{") - (s[k] == "}")
        if depth == 0:
            return k + 1
    raise AssertionError("unbalanced braces")


def _functions():
    """(name, head, body, is kernel) of every device function and kernel."""
    out = []
    for path in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]):
        s = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__|__device__", s):
            i = re.compile(r"[{;]").search(s, m.end())
            if not i or s[i.start()] == ";":
                continue
            head = s[m.end():i.start()]
            head = re.sub(r"__launch_bounds__\([^\n]*?\)\)?(?=\s)", "", head)
            names = re.findall(r"([A-Za-z_]\w*)\s*\(", head)
            if names:
                names = [n for n in names if n not in ("__launch_bounds__", "__align__")]
                out.append((names[0], head, s[i.start():_block(s, i.start())], m.group(0) == "__global__"))
    return out


def _reached(name, functions, seen):
    for n, head, body, _ in functions:
        if n == name and (n, head) not in seen:
            seen[(n, head)] = body
            for callee in set(re.findall(r"([A-Za-z_]\w*)\s*(?:<[^;(){}]*>)?\s*\(", body)):
                _reached(callee, functions, seen)
    return seen


def test_dependent_kernels_read_by_plain_loads():
    functions = _functions()
    kernels = [f for f in functions if f[3]]
    assert len(kernels) > 40
    waiting, faults = [], []
    for name, head, body, _ in kernels:
        bodies = _reached(name, functions, {})
        if not any(WAIT.search(b) for b in bodies.values()):
            continue
        waiting.append(name)
        allowed = COMPLETE.get(name, set())
        for p in re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", head):
            if p not in allowed:
                faults.append(f"{name}: const __restrict__ {p}")
        for (fn, _h), b in bodies.items():
            b = GUARDED.sub("", b)
            for arg in re.findall(r"__ldg\(\s*(?:reinterpret_cast<[^>]*>\()?\s*(\w+)", b):
                if arg not in allowed:
                    faults.append(f"{name}: __ldg({arg}) in {fn}")
    told = {}
    for name, head, body, _ in functions:
        for use in re.findall(r"stage_tiles<\d, true>|TileView<true>|load<true>", head + body):
            told.setdefault(name, set()).add(use)
    assert told == TOLD
    assert len(waiting) >= 35, waiting
    assert not faults, "\n".join(sorted(set(faults)))
