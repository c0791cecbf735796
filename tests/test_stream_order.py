"""The context's device memory is cleared on the context's own stream.  The
stream does not wait for the default stream (cudaStreamNonBlocking), so a plain
cudaMemset could still be under way when a kernel of the context reads."""

import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_context_memory_is_cleared_on_its_stream():
    with open(os.path.join(ROOT, "ggems_b200", "csrc", "gg_runtime.cu")) as f:
        text = f.read()
    assert "cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking)" in text
    assert len(re.findall(r"cudaMemsetAsync\([^;]*c->stream\)", text)) > 10
    assert not re.findall(r"\bcudaMemset\(", text)
