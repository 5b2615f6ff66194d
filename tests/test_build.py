"""Which sources the build compiles in parts (--split-compile changes the generated code)."""
import glob
import os

from fhe_b200 import build


def test_only_the_transforms_are_compiled_in_parts():
    sources = [os.path.basename(f) for f in glob.glob(os.path.join(build.CSRC, "*.cu"))]
    assert {"bsgs.cu", "kernels.cu", "moddown_tc.cu", "modup_tc.cu", "rotate.cu"} < set(sources)
    split = {f for f in sources if any("split-compile" in a for a in build.arch_flags(f))}
    assert split == set(build.SPLIT_COMPILED)
    assert all(f.startswith("ntt_") and f != "ntt_tc.cu" for f in split)
