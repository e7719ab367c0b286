"""Order of the library's own copies and fills against its kernels (CPU: reads the sources).

Handles and preconditioners run on non-blocking streams, which do not wait for the legacy default stream.
cudaMemcpy from pageable memory may return while the bytes are only staged, and cudaMemset returns at
once, so a kernel launched behind either could read the old bytes -- an offset list, for one, that it
writes through.  Host-to-device copies and fills therefore name the stream of the kernels that follow."""
import glob
import os
import re

import pytest

from conftest import ROOT

SOURCES = sorted(glob.glob(os.path.join(ROOT, "sbd-pub_b200", "csrc", "*.cu*")))


def _calls(text, name):
    """The argument texts of every call of `name`."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"\b%s\s*\(" % name, text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        yield text[m.end():i - 1]


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_uploads_and_fills_name_their_stream(path):
    text = open(path).read()
    assert not [a for a in _calls(text, "cudaMemcpy") if "HostToDevice" in a or "Default" in a]
    assert not list(_calls(text, "cudaMemset"))
    for a in _calls(text, "cudaMemcpyAsync"):
        assert re.search(r"\b(\w+->)?st(ream)?$", a.rsplit(",", 1)[1].strip()), a
