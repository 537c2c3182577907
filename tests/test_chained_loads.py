"""The load rule of chained kernels (csrc/common.cuh, chain()), on their source: a kernel whose CTAs may be resident
while the one before it in the stream still runs reads what the chain writes with ld_chain, or plainly through a pointer
that is not const __restrict__. What may be read otherwise is complete before the chain's first kernel starts, and is
named here, kernel by kernel."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "ray-tracer_gb300" / "csrc"

# pointers to what no kernel of the chain writes (hist in k_sort_hist: its own CTAs' sums, read past the L1)
COMPLETE = {
    "k_sort_hist": {"keys", "q", "hist", "d_count"},
    "k_onesweep": {"d_count"},
    "k_compress_write": {"keys"},
    "k_dc_write": {"counts"},
    "k_dc_expand": {"counts", "skeys", "trimmed", "po"},
    "k_fused_rays": {"tris", "nodes", "ent"},  # the scene
}


def _close(s: str, i: int, pair: str) -> int:
    """The index past the bracket that closes the one at s[i]."""
    depth = 0
    for k in range(i, len(s)):
        depth += (s[k] == pair[0]) - (s[k] == pair[1])
        if depth == 0:
            return k + 1
    raise AssertionError("unbalanced source")


def _functions(text: str, head: str):
    """(name, parameters, body) of the functions whose definition starts with `head`."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(head, text):
        d = re.compile(r"\b(?!__launch_bounds__)(\w+)\s*\(").search(text, m.end())
        p1 = _close(text, d.end() - 1, "()")
        if text[p1:].lstrip()[:1] == "{":
            b0 = text.index("{", p1)
            yield d.group(1), text[d.end():p1], text[b0:_close(text, b0, "{}")]


def _chained():
    for f in sorted(CSRC.glob("*.cu")):
        for name, params, body in _functions(f.read_text(), r"__global__\s+void\s"):
            if "griddepcontrol.wait" in body or re.search(r"\bchain\(\);", body):
                yield name, params, body


KERNELS = {name: (params, body) for name, params, body in _chained()}


def test_the_chained_kernels_are_found():
    assert {"k_onesweep", "k_bounce", "k_fused_rays", "k_dc_expand", "k_ploc_pass", "k_level_cuts"} <= set(KERNELS)


@pytest.mark.parametrize("name", sorted(KERNELS))
def test_no_read_only_load_of_what_the_chain_writes(name):
    params, body = KERNELS[name]
    ok = COMPLETE.get(name, set())
    for m in re.finditer(r"\b(__ldg|__ldcg|load_ray)\(", body):
        arg = body[m.end():_close(body, m.end() - 1, "()")]
        assert set(re.findall(r"\w+", arg)) & ok, f"{name}: {m.group(0)}{arg}"
    for p in re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", params):
        if p not in ok:
            assert not re.search(rf"\b{p}\s*\[|\*\s*{p}\b", body), f"{name}: plain read through const __restrict__ {p}"


def test_shading_reads_shadow_flags_by_the_rule():
    """k_bounce calls shade_surface behind the launch that writes the flags."""
    fns = {n: (p, b) for n, p, b in _functions((CSRC / "pixel.cuh").read_text(), r"RSH_DEV void ")}
    params, body = fns["shade_surface"]
    assert not re.search(r"__restrict__\s+shadow", params) and "__ldg" not in body


def test_the_second_of_a_pair_acquires_before_it_reads():
    """k_fused_rays as the second launch of a frame's pair does not wait for the first, so what the kernel before both
    wrote (lists, counts, rays) is visible to it only through the word that the first releases after its own wait."""
    body = KERNELS["k_fused_rays"][1]
    wait, release = body.index("griddepcontrol.wait"), body.index("st_release_u32(a.ready")
    acquire, trigger = body.index("ld_acquire_u32(a.ready)"), body.index("griddepcontrol.launch_dependents")
    assert wait < release < trigger and acquire < trigger < body.index("dev_count(")
    spin = body[body.rindex("for (", 0, acquire):trigger]
    assert "RSH_SPIN_LIMIT" in spin and "raise_device_error" in spin  # the wait ends, with an error
    frame = (CSRC / "engine.cu").read_text()
    assert len(re.findall(r"trace_alone\([^;]*\btrue, ready\)", frame)) == 2  # both launches of a frame's pair
