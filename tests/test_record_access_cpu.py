"""The records' 256-bit loads and stores and the copies into shared memory are
inline assembly, so the compiler knows that they touch memory only from their clobber; the batch kernel stores
values in one phase that it loads so in a later one.  Read from the source,
since a wrong order need not show in a run."""
import glob
import os
import re

from fdm_cell_based_amr_cartesian_b200 import build as B


def test_assembly_on_global_memory_says_so():
    seen = 0
    for path in glob.glob(os.path.join(B.CSRC, "*.cu*")):
        txt = re.sub(r"//[^\n]*", "", open(path).read())
        for a in re.findall(r"\basm\b[^;]*?\((?:[^;\"]|\"[^\"]*\")*\);", txt):
            if re.search(r'"(ld\.global|st\.global|cp\.async)', a):
                seen += 1
                assert "volatile" in a and '"memory"' in a, (os.path.basename(path), a)
    assert seen >= 5
