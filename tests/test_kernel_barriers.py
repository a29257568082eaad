"""The four-warp Newmark kernel's barriers, read from its source (a block barrier in
conditional code is undefined wherever it seems to work, so no run shows it): every
__syncthreads() is a statement of the kernel's own body, under no condition and in no
lambda, and the barrier at which warps meet at different places has a stated count that
its participants add up to."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "muscade.jl_gb300", "csrc", "mgpu.cu")


def _body(text, name):
    at = text.index("{", text.index(")", text.index(name + "(int64_t")))
    depth = 0
    for k in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[k], 0)
        if depth == 0:
            return text[at + 1 : k]


def test_block_barriers_stand_outside_every_condition():
    body = re.sub(r"//[^\n]*", "", _body(open(SRC).read(), "beam_split_kernel"))
    at = [m.start() for m in re.finditer(r"__syncthreads\(\)", body)]
    assert at
    for k in at:
        head = body[:k]
        assert head.count("{") == head.count("}"), "a block barrier inside a block or lambda"
        assert head.rstrip()[-1] in ";}", "a block barrier under a condition"
    counted = re.findall(r"barrier\.cta\.(arrive|sync) (\d+), (\d+);", body)
    assert sorted(kind for kind, _, _ in counted) == ["arrive", "sync"]
    assert {(b, n) for _, b, n in counted} == {("1", "96")}  # the three column warps
