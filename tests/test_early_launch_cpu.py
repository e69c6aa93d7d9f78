"""Kernels that are launched before their predecessor has ended wait before they
touch global memory.

What earlier kernels of a stream wrote is promised to be visible to a kernel
that has executed griddepcontrol.wait, not to one that started early; no run
can show that a missing wait does no harm.  So the order is checked in the
source: in the body of every kernel that is launched early, the first
unconditional pdl_wait (or pdl_sync) comes before any access through a pointer
of the kernel's arguments."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "tfg_b200" / "csrc"

# an argument array indexed, dereferenced or handed on: a.state[...], *a.loss, train_navail(a)
TOUCH = re.compile(r"\ba\.[\w.]+\s*\[|(?:[=(,;]|return)\s*\*\s*a\.\w|\btrain_navail\(|\ba\.ws\.|\bload_aprims_smem\(|__ldg\(|bulk_g2s\(")


def _body(src: str, kernel: str) -> str:
    """The kernel's body, from its opening brace to the brace in column 0."""
    m = re.search(r"__global__[^;{]*\b%s\([^)]*\)\s*\{\n" % kernel, src)
    assert m, kernel
    return src[m.end():src.index("\n}\n", m.end())]


def _touched_before_wait(body: str, wait: str) -> list[str]:
    seen = []
    for line in body.splitlines():
        code = line.split("//")[0]
        if re.match(r"    %s\(\);" % wait, code):   # unconditional: a statement of the body itself
            return seen
        seen += TOUCH.findall(code)
    return seen + ["no unconditional %s()" % wait]


@pytest.mark.parametrize("kernel", ["k_train", "k_train128", "k_wgrad", "k_adam", "k_adam_hash"])
def test_training_kernels_wait_first(kernel):
    src = (CSRC / "nrc_mlp.cu").read_text()
    assert "launch_early(mlp::%s" % kernel in src
    assert _touched_before_wait(_body(src, kernel), "pdl_wait") == []


def test_no_other_training_kernel_is_launched_early():
    src = (CSRC / "nrc_mlp.cu").read_text()
    names = set(re.findall(r"launch_early\(mlp::(\w+)", src))
    assert names == {"k_train", "k_train128", "k_wgrad", "k_adam", "k_adam_hash"}


@pytest.mark.parametrize("kernel,wait", [("k_shade", "pdl_sync"), ("k_resolve", "pdl_sync"), ("k_trace", "pdl_wait")])
def test_render_kernels_wait_first(kernel, wait):
    assert _touched_before_wait(_body((CSRC / "render.cu").read_text(), kernel), wait) == []


def test_short_queue_kernel_waits_or_acquires_first():
    src = (CSRC / "render.cu").read_text()
    body = _body(src, "k_few")
    head, rest = body.split("    if (always) {\n", 1)
    assert TOUCH.findall(head) == [] and rest.lstrip().startswith("pdl_sync();")
    beside = rest.split("    } else {", 1)[1].split("    }\n", 1)[0]
    assert "handed_over(" in beside.split(";")[0]
    # the length comes with acquire semantics, or after a wait; it was released before k_few could start
    take = src[src.index("uint32_t handed_over("):]
    take = take[:take.index("\n}\n")]
    assert take.index("ld.acquire.gpu") < take.index("pdl_wait();") < take.index("return counters[")
    give = src[src.index("void hand_over("):]
    give = give[:give.index("\n}\n")]
    assert give.index("st.release.gpu") < give.index("__syncthreads();") < give.index("pdl_launch();")
    for kernel in ("k_trace", "k_shadow"):
        assert "pdl_launch" not in _body(src, kernel) and "hand_over(" in _body(src, kernel)


def test_no_other_render_kernel_is_launched_early():
    src = (CSRC / "render.cu").read_text()
    assert set(re.findall(r"[ (]launch\((\w+)<", src)) == {"k_few", "k_shade", "k_resolve", "k_trace"}
