"""The blocks of a cluster send sums into one another's shared memory.  A block ends by itself only when all that is sent to it has come; one whose wait ran
out has to stay until nobody can send any more, and no block may end while copies of its own are on their way to its shared memory.  Read from the sources."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "poptransformer_b200", "csrc")


def _text(name):
    return re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())


def _kernel(text, start):
    """The body of the kernel whose declaration contains `start`."""
    i = text.index("{", text.index(")", text.index(start)))
    depth = 0
    for j in range(i, len(text)):
        depth += (text[j] == "{") - (text[j] == "}")
        if depth == 0:
            return text[i:j + 1]


def test_meeting_has_all_threads_and_ends():
    text = _text("mbarrier.cuh")
    body = _kernel(text, "void stay_for_cluster(")
    assert body.index("__syncwarp()") < body.index("barrier.cluster.arrive.release.aligned") < body.index("barrier.cluster.wait.acquire.aligned")
    assert "WAIT_LIMIT" in _kernel(text, "void mbar_wait_ring(")


def test_attention():
    body = _kernel(_text("attention.cu"), "kv_append_attn_kernel(")
    failed = re.search(r"if \(!__all_sync\(0xffffffffu, mbar_wait\(arrived, 0, &sm\.abort\)\)\) \{(.*?)\}", body, re.S)
    assert failed and "stay_for_cluster();" in failed.group(1)          # (the whole warp decides: the meeting wants whole warps)
    assert len(re.findall(r"mbar_wait\(", body)) == 1


def test_few_rows():
    text = _text("gemm_few.cu")
    body = _kernel(text, "linear_kernel(const Params")
    assert re.search(r"if \(slices > 1 && __any_sync\(0xffffffffu, ctl\.abort\)\) stay_for_cluster\(\);", text)
    for m in re.finditer(r"\breturn;", body):                            # every way out between the first send and the end
        assert "leave(ctl, slices);" in body[:m.start()].splitlines()[-1] + body[:m.start()].splitlines()[-2], body[m.start() - 200:m.start()]
    asked = body[body.index("bulk_g2s("):]
    assert asked.index("mbar_wait_ring(full0, st, S)") < asked.index("return;")
    assert body.index("cp.async.wait_all") < body.index("return;")


@pytest.mark.parametrize("kernel", ["gemm_dense_kernel(", "gemm_int4_kernel("])
def test_tensor_memory_products(kernel):
    text = _text("gemm_tc.cu")
    body = _kernel(text, kernel)
    end = body[body.rindex("__syncthreads();"):]                         # nobody gives up behind this: all threads go the same way
    assert "give_up" not in end and end.index("if (ctl.abort) end_after_failure(") < end.index("tmem_dealloc")
    closing = _kernel(text, "void end_after_failure(")
    assert "mbar_wait_ring(full0, issued, stages)" in closing and "mbar_wait_ring(sa(&ctl.accum), 1, 1)" in closing
    assert closing.index("if (ksplit > 1) stay_for_cluster();") < closing.index("__syncthreads();")
    asks = re.findall(r"give_up\(ctl, p\.error_flag, 2[15]\); break; \}\s*issued = it \+ 1;", body)     # what was asked for is counted, also where the loop breaks off
    assert len(asks) == len(re.findall(r"give_up\(ctl, p\.error_flag, 2[15]\); break;", body)) >= 1
