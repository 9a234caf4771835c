"""Results that a kernel leaves in host memory beside the number of their call (mul_mat of host pointers)."""
import glob
import os
import re

import gemma_ggml_b200 as G

CSRC = os.path.join(os.path.dirname(G.CUDA_LIB), "csrc")


def test_a_word_for_another_processor_is_one_scalar_store():
    """Numbers that belong together, payload and tag, arrive together only where one scalar store of eight bytes writes them: the numbers of a vector store are
    stores of their own, in no stated order."""
    found = 0
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        for m in re.finditer(r'"(st\.[\w.:]*\bsys\b[\w.:]*)', open(path).read()):
            found += 1
            assert re.search(r"\.[bu]64$", m.group(1)) and not re.search(r"\.v[248]\b", m.group(1)), (path, m.group(1))
    assert found >= 2
