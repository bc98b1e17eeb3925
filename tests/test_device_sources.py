"""CPU checks of what the device code's correctness rests on but no result can
show on a given GPU: read from the sources."""
import os
import re

import x2dhf_gb300 as xg

CSRC = os.path.join(os.path.dirname(xg.__file__), "csrc")


def _functions(name):
    """name -> body of the small device functions of a source file."""
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    found = re.findall(r"__device__ __forceinline__ \w+ (\w+)\([^)]*\) \{\n(.*?)\n\}", text, re.S)
    return dict(found)


def test_tagged_words_are_read_and_written_whole():
    """The FP64 sweeps without barriers hand a value over together with its
    tag, with no other ordering: every load and store of such a word is one
    128-bit scalar access (single-copy atomic), in global and in shared
    memory.  A vector of two 64-bit accesses may be taken apart."""
    fn = _functions("x2g_kernels.cu")
    for name, op, space in (("ld_tagged", "ld.relaxed.gpu", "global"), ("st_tagged", "st.relaxed.gpu", "global"),
                            ("ld_near", "ld.relaxed.cta", "shared"), ("st_near", "st.relaxed.cta", "shared")):
        assert f"{op}.{space}.b128" in fn[name], name
        assert ".v2." not in fn[name] and "volatile." not in fn[name], name
