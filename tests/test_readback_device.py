"""The read-backs of sites pack them in a kernel on the engine's stream, which
CUDA refuses while another device is current; as plain copies they worked from
any device.  One GPU cannot show that, so the source is read: an entry point
that only reads state back and launches a kernel makes the engine's device
current first, and gives the caller's back."""
import re

from conftest import PKG_DIR


def body(src, name):
    start = re.search(r"^int %s\(.*?\) \{$" % name, src, re.M).end()
    return src[start:src.index("\n}\n", start)]


def test_readbacks_launch_on_the_engines_device():
    src = (PKG_DIR / "csrc" / "engine.cu").read_text()
    readers = re.findall(r"^int (vgb_engine_(?:get|copy)_\w+)\(", src, re.M)
    assert {"vgb_engine_get_sites", "vgb_engine_get_sites_original"} <= set(readers)
    for name in readers:
        b = body(src, name)
        if "<<<" in b:
            assert "const OnDevice on(e->cfg.device);" in b[:b.index("<<<")], name
    guard = src[src.index("struct OnDevice {"):]
    guard = guard[:guard.index("\n};")]
    assert guard.count("cudaSetDevice(") == 2 and "cudaSetDevice(back)" in guard
