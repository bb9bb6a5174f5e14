"""Kernel-trace ids: a file tag names one source file, the one the reader of a trace is told."""
import os
import re

import batchgen_b200
from batchgen_b200.utils import kernel_trace

PKG = os.path.dirname(batchgen_b200.__file__)


def test_file_tags_are_unique_and_known():
    tags = {}
    for d in ("ops/csrc", "parallel/csrc"):
        for name in sorted(os.listdir(os.path.join(PKG, d))):
            if name.endswith(".cu"):
                m = re.search(r"^#define BG_FILE_TAG (\d+)", open(os.path.join(PKG, d, name)).read(), re.M)
                if m:
                    tags.setdefault(int(m.group(1)), []).append(f"{d}/{name}")
    assert all(len(files) == 1 for files in tags.values()), tags
    for tag, path in kernel_trace.FILES.items():
        if path.endswith(".cu"):
            assert tags[tag] == [path]
