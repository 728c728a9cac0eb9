"""Uploads are ordered before the kernels that read them. The engine's streams are non-blocking, so they do not wait for
the default stream, and a blocking copy from pageable memory may return before the data has arrived: every upload and
clearing of device memory names the stream it goes on."""
import os
import re

import pytest

CUDA = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "csu_b200", "csrc", "cuda")


def _calls(src, name):
    for m in re.finditer(r"\b%s\(" % name, src):
        depth, k = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(src[k], 0)
            k += 1
        yield src[m.start():k]


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CUDA) if f.endswith(".cu")))
def test_no_upload_on_the_default_stream(name):
    src = open(os.path.join(CUDA, name)).read()
    assert not [c for c in _calls(src, "cudaMemcpy") if "HostToDevice" in c]
    assert not list(_calls(src, "cudaMemset"))
