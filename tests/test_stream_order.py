"""Every device copy and clear of the library is issued on one of the context's streams.  These do not wait for the default stream,
so a table copied or cleared there could still be on its way when a kernel reads it."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_no_default_stream_copies():
    found = []
    for f in sorted(glob.glob(os.path.join(ROOT, "eom-imsrg_gb300", "csrc", "*"))):
        text = re.sub(r'"(\\.|[^"\\])*"', '""', re.sub(r"//[^\n]*", "", open(f).read()))
        found += [(os.path.basename(f), m.group(0)) for m in re.finditer(r"\bcuda(Memcpy|Memset|Memcpy2D|MemcpyToSymbol)\s*\(", text)]
    assert not found, found
