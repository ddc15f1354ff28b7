"""Inputs of a launch are copied on the stream of the launch: the library's streams do
not block on the default stream, and a copy there from pageable memory may return
before its data has reached the device."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lair_gb300", "csrc")


def test_no_copies_to_the_device_on_the_default_stream():
    found = []
    for name in sorted(os.listdir(CSRC)):
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read()) if name.endswith((".cu", ".cuh")) else ""
        for call in re.findall(r"\bcudaMem(?:cpy|set|cpy2D)\s*\([^;]*;", text):
            if "cudaMemcpyDeviceToHost" not in call:
                found.append((name, call))
    assert not found
