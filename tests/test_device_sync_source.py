"""Rules of the device code's synchronisation that no run shows: a GPU does what
one expects when they are broken, until it does not.  Read from the sources."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "product-graph-cycles_b200", "csrc")


@pytest.fixture(scope="module")
def functions():
    """Body of every function of the Bellman-Ford sources, comments removed."""
    out = {}
    for name in ("kernels_bf.cu", "bf_local.cuh"):
        with open(os.path.join(CSRC, name)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for m in re.finditer(r"^(?!\s|#|template|struct|namespace|using|constexpr|static_assert|extern)[^;={}]*?(\w+)\([^{};]*\)\s*\{\n",
                             text, re.M):
            end = text.index("\n}", m.end() - 1)
            out[m.group(1)] = text[m.end():end]
    return out


def _callers(functions, name):
    return {f for f, body in functions.items() if re.search(r"\b%s\s*[<(]" % name, body)}


def test_an_mbarrier_ends_before_its_words_are_used_again(functions):
    """Every mbarrier.init belongs to a Bellman-Ford call that invalidates both
    words after its last use (a launch makes many calls)."""
    assert {f for f, body in functions.items() if "mbarrier.init." in body} == {"mbar_init"}
    assert _callers(functions, "mbar_init") == {"bf_run", "local_begin"}
    assert _callers(functions, "local_begin") == {"bf_run"}
    assert _callers(functions, "bf_run") == {"bf_body"}
    body = functions["bf_body"]
    after = body[body.index("bf_run<"):]
    assert re.search(r"__syncthreads\(\);.*mbar_inval\(bar\);.*mbar_inval\(bar \+ 1\);.*__syncthreads\(\);", after, re.S)
    assert "mbarrier.inval.shared::cta.b64" in functions["mbar_inval"]


def test_a_cta_leaves_a_step_as_one(functions):
    """The error word of a team is written by other CTAs at any time: the
    threads of a CTA that read it one by one may disagree, and part of them
    would miss the next barrier."""
    body = functions["step_handoff"]
    assert re.search(r"return sGood != 0;\s*$", body)
    assert re.search(r"if \(threadIdx\.x == 0\) \{[^{}]*sGood = good;\s*\}", body)
    assert "const int raised = *(volatile int*)t.err;" in body
    assert "good = !__any_sync(0xffffffffu, raised != 0);" in body
    assert body.count("t.err") == body.count("atomicExch(t.err, 1)") + 1


def test_exchanged_records_are_overwritten_after_their_reads(functions):
    """A CTA's report that it has read its neighbours' records (stepDone) is
    the only order between those reads and the stores that replace the records:
    release and acquire, each beyond a CTA barrier."""
    body = functions["local_sweep"]
    assert re.search(r"__syncthreads\(\);\s*if \(lane == 0 && [^{}]*\)\s*st_release_u32\(H\.stepDone", body)
    assert "while ((int)ld_acquire_u32(f) < want)" in body
    assert len(re.findall(r"H\.stepDone", body)) == 2
    for f, b in functions.items():
        assert "relaxed.gpu.global.u32" not in b, f
    assert "st.release.gpu.global.u32" in functions["st_release_u32"]
    assert "ld.acquire.gpu.global.u32" in functions["ld_acquire_u32"]
