"""Orders that the kernels' sources have to keep and that no run shows reliably:
each rule is read off the text of the kernels it is about."""
import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "aquarius_b200" / "csrc"
SOURCES = {p.name: p.read_text() for p in sorted(CSRC.glob("*.cu*"))}


def _code(text):
    return re.sub(r"//[^\n]*", "", text)


def _kernels(text):
    """(name, body) of every __global__ function definition."""
    out = []
    for m in re.finditer(r"__global__\s+void[^;{]*?\b(k\w+)\s*\(", text):
        at = text.index(")", m.end())
        brace, semi = text.find("{", at), text.find(";", at)
        if brace < 0 or 0 <= semi < brace:
            continue  # a declaration
        depth, i = 0, brace
        while True:
            depth += (text[i] == "{") - (text[i] == "}")
            i += 1
            if depth == 0:
                break
        out.append((m.group(1), text[brace:i]))
    return out


KERNELS = {f"{f}:{name}": body for f, text in SOURCES.items() for name, body in _kernels(_code(text))}


@pytest.mark.parametrize("kernel", [k for k, b in KERNELS.items() if "griddepcontrol.launch_dependents" in b])
def test_a_first_launch_waits_before_it_triggers(kernel):
    """A kernel that triggers its dependents has a path, ahead of the trigger,
    that has waited for its own predecessor: the first launch of a chain takes
    it, so what later launches read early was complete before they started."""
    body = KERNELS[kernel]
    assert 0 <= body.find("griddepcontrol.wait") < body.find("griddepcontrol.launch_dependents")


@pytest.mark.parametrize("array", ["umap", "list", "part", "pa"])
def test_cluster_solve_reads_what_it_writes_through_l2(array):
    """The cluster solve's CTAs exchange these arrays within one launch: the
    read-only path (__ldg) is for data that stays constant for a kernel's life."""
    code = _code(SOURCES["k_cluster.cu"])
    assert re.search(rf"\bS\.{array}\b", code)
    assert not re.search(rf"__ldg\(\s*S\.{array}\b", code)


@pytest.mark.parametrize("kernel", [k for k, b in KERNELS.items() if "mbar_wait(" in b])
def test_bounded_waits_are_decided_by_whole_warps(kernel):
    """A wait that may run out for some lanes alone must not steer a warp around
    tcgen05.ld, which all of its lanes execute together."""
    body = KERNELS[kernel]
    assert "mbar_wait(" not in re.sub(r"__all_sync\(0xffffffffu, mbar_wait\(", "", body)


def test_dependent_mmas_share_accumulator_and_shape():
    """tcgen05.mma instructions are ordered among themselves only with the same
    accumulator and shape.  The convolution issues one form of it per halo
    plane, and a plane's after those of the plane before have completed."""
    body = KERNELS["k_unet.cu:k_conv3_fwd_umma"]
    assert body.count("umma_f16(") == 1
    issue = body.index("umma_f16(")
    assert body.rfind("wait_plane(h - 1)", 0, issue) > body.rfind("__syncthreads_and", 0, issue) > 0


def test_splat_leaves_by_a_vote():
    """Other CTAs set the flag that ends the counting: its value may differ from
    thread to thread, so the CTA leaves on one thread's reading, together."""
    body = KERNELS["k_render.cu:k_phase_splat"]
    assert "return" not in body[:body.index("__syncthreads")]
    for m in re.finditer(r"__ldcg\(mixed\)", body):
        assert re.search(r"__syncthreads_or\(tid == 0 && $", body[:m.start()])


@pytest.mark.parametrize("source", [f for f, t in SOURCES.items() if "cudaFuncSetAttribute" in t])
def test_kernel_attributes_are_set_on_every_device(source):
    """cudaFuncSetAttribute acts on the current device: its result is not kept in
    a static of the process."""
    assert not re.search(r"static\s+(const\s+)?cudaError_t\s+\w+\s*=", _code(SOURCES[source]))
