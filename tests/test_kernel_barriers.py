"""Orderings that a kernel's source has to show, because a run that breaks one
may still give the right result: read from the source, without a GPU.

A CTA of a cluster may touch another CTA's shared memory only once that CTA runs
and while it has not left: a cluster barrier before the first remote access and
one after the last."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "tailor_gb300" / "csrc"


def kernels(text):
    """(name, body) of every __global__ function, without comments."""
    text = re.sub(r"//[^\n]*", "", text)
    out = []
    for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\(", text):
        at = text.index("{", m.end())
        depth, end = 0, at
        while True:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
            if depth == 0:
                break
        out.append((m.group(1), text[at:end]))
    return out


CLUSTER = [(name, body) for f in sorted(CSRC.glob("*.cu"))
           for name, body in kernels(f.read_text()) if "map_shared_rank" in body
           or "cluster_argmax" in body]


def test_the_cluster_kernels_are_found():
    assert {n for n, _ in CLUSTER} == {"k_panel_cluster", "k_panel_cluster_sm"}


@pytest.mark.parametrize("name,body", CLUSTER, ids=[n for n, _ in CLUSTER])
def test_remote_accesses_lie_between_cluster_barriers(name, body):
    # names of pointers into another CTA, then every place that goes through one
    remote = re.findall(r"\*(\w+) = cluster\.map_shared_rank\(", body)
    uses = [m.start() for m in re.finditer(r"\*cluster\.map_shared_rank\(|cluster_argmax<", body)]
    for v in remote:
        uses += [m.start() for m in re.finditer(rf"\b{v}\[", body)]
    syncs = [m.start() for m in re.finditer(r"cluster\.sync\(\)", body)]
    assert uses and syncs
    assert syncs[0] < min(uses), "a remote access before the first cluster barrier"
    assert syncs[-1] > max(uses), "a remote access after the last cluster barrier"


WARP_ROLE = re.compile(r"\(warp == (\d+)\) \{")
FULL_MASK = re.compile(r"__\w+_sync\(|__syncwarp\(")


def block(text, at):
    """The braces' contents from the { at or after `at`, and their end."""
    at = text.index("{", at)
    depth, end = 0, at
    while True:
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        end += 1
        if depth == 0:
            return text[at + 1:end - 1], end


def one_lane_only(body):
    """The parts of a warp's code that stand under if (lane == 0)."""
    out = []
    for m in re.finditer(r"if \(lane == 0\)\s*", body):
        if body[m.end()] == "{":
            end = block(body, m.end())[1]
        else:
            end = body.index(";", m.end()) + 1
        out.append((m.end(), end))
    return out


def test_a_whole_warp_leaves_together():
    """A role whose warp works as a whole (full-mask shuffles, reductions or
    barriers) reads the abort word in its first lane only and passes it on: lanes
    that read it each for themselves could leave one by one, and the others would
    wait for them at the next full-mask operation."""
    found = 0
    for f in sorted(CSRC.glob("*.cu")):
        for name, body in kernels(f.read_text()):
            if "abort_flag" not in body:
                continue
            for m in WARP_ROLE.finditer(body):
                role, _ = block(body, m.end() - 1)
                lanes = one_lane_only(role)
                inside = lambda at: any(a <= at < b for a, b in lanes)  # noqa: E731
                if not any(not inside(x.start()) for x in FULL_MASK.finditer(role)):
                    continue  # one lane does everything
                for r in re.finditer(r"abort_flag|wait_bar\(", role):
                    found += 1
                    assert inside(r.start()), f"{name}: warp {m.group(1)}"
    assert found
