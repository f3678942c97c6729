"""Rules of the tensor-core and path kernels whose breach no run shows reliably (it would hang or
race on some machine, some day), checked on their source: which lanes may wait or store where, and
in which order a kernel takes resources. Comments are stripped before reading."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "kuafu_gb300" / "csrc"


def _source(name):
    s = (CSRC / name).read_text()
    s = re.sub(r"/\*.*?\*/", "", s, flags=re.S)
    return re.sub(r"//[^\n]*", "", s)


def _body(s, at):
    """The brace block that opens at or after position `at`, without its braces."""
    i = s.index("{", at)
    depth, j = 0, i
    while True:
        depth += {"{": 1, "}": -1}.get(s[j], 0)
        if depth == 0:
            return s[i + 1:j]
        j += 1


def _function(s, name):
    """The body of the function defined as `name` (the match whose parameter list a block follows)."""
    for m in re.finditer(r"\b" + name + r"\s*\(", s):
        depth, j = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(s[j], 0)
            j += 1
        if re.match(r"\s*\{", s[j:]):
            return _body(s, j)
    raise AssertionError(f"no definition of {name}")


def _kernels(s):
    names = re.findall(r"__global__\s+void\s+(?:__launch_bounds__\s*\([^()]*(?:\([^()]*\)[^()]*)*\)\s*)?(\w+)\s*\(", s)
    return {n: _function(s, n) for n in names}


def _headers_at(body, at):
    """What opens each block around position `at`: the text before its brace."""
    stack, start = [], 0
    for i, c in enumerate(body[:at]):
        if c == "{":
            stack.append(body[start:i])
        elif c == "}":
            stack.pop()
        if c in "{};":
            start = i + 1
    return stack


CONV = _kernels(_source("kf_conv.cu"))


def test_the_kernels_are_found():
    assert {"k_tc", "k_conv_halo", "k_conv_tile", "k_wgrad"} <= set(CONV)


@pytest.mark.parametrize("kernel", sorted(CONV))
def test_a_warp_waits_and_gives_up_as_one(kernel):
    """A bounded wait that each lane decides for itself stands only where a single lane runs: a warp
    whose lanes disagree would run TMEM loads and shuffles with a part of its lanes."""
    body = CONV[kernel]
    for m in re.finditer(r"\bmbar_wait\s*\(", body):
        headers = _headers_at(body, m.start())
        assert any("lane == 0" in h or "threadIdx.x == 0" in h for h in headers), body[m.start():m.start() + 80]


@pytest.mark.parametrize("kernel", sorted(k for k in CONV if "tmem_alloc" in CONV[k]))
def test_tmem_is_held_before_the_next_kernel_may_start(kernel):
    """A kernel that may start early takes TMEM before it waits for the one ahead: had that one not
    allocated yet, both would wait for each other, and a TMEM allocation waits without a bound."""
    body = CONV[kernel]
    triggers = [m.start() for m in re.finditer(r"\bgrid_(dependency_wait|launch_dependents)\s*\(", body)]
    assert all(t > body.index("tmem_alloc(") for t in triggers)


def _calls(body, name):
    """The arguments of each call of `name` in a body, as one string without line breaks."""
    for m in re.finditer(r"\b" + name + r"<\w+>\s*\(", body):
        depth, j = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(body[j], 0)
            j += 1
        yield " ".join(body[m.end():j - 1].split())


def test_one_lane_of_a_shared_path_writes_its_aovs():
    """Several lanes may run one path: what clears a pixel's AOVs or writes them does it in the
    path's first lane, so that no lane that falls behind clears what another has written."""
    body = _kernels(_source("kf_wavefront.cu"))["k_paths"]
    for name in ("camera_path", "miss_emission", "shade_hit"):
        calls = list(_calls(body, name))
        assert calls and all("sub == 0" in c for c in calls), name
    for m in re.finditer(r"w\.(radiance|primary|albedo|normal|depth|seg)\[[^\]]*\]\s*=[^=]", body):
        line = body[body.rindex("\n", 0, m.start()):m.start()]
        assert any("sub == 0" in h for h in _headers_at(body, m.start()) + [line]), m.group(0)


def test_captured_launches_are_known_by_all_of_the_wavefront_state():
    """A captured launch sequence bakes in the wavefront state by value. Its key takes every byte of
    it: with a few addresses only, a replay could read buffers that were freed since (an allocator
    may return one of them to its old place and not the others)."""
    s = _source("kf_render.cu")
    assert "sizeof(w)" in _function(s, "wave_key")
    for f in ("render_frame", "render_batch"):
        (key,) = re.findall(r"std::string key = ([^;]*);", _function(s, f))
        assert "wave_key(w)" in key
