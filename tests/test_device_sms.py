"""The launch rules count the SMs of the device they run on: no kernel source repeats the number
of one card beside the query."""
import glob
import os
import re

from conftest import PKG


def test_rules_ask_the_device_for_its_sms():
    for path in sorted(glob.glob(os.path.join(PKG, "csrc", "*"))):
        text = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)
        found = re.findall(r"[^\n]*\b(?:152|304|608)\b[^\n]*", text)
        # the value taken where the query fails
        assert all("cudaDevAttrMultiProcessorCount" in line for line in found), (os.path.basename(path), found)
