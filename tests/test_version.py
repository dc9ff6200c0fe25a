"""The library version tells callers of grass_device_view which layout they get."""
import re

import grass_b200 as G


def test_version_names_the_layout():
    version = re.fullmatch(rb"grass_b200 (\d+\.\d+) \(sm_100a\)", G.lib.grass_version()).group(1).decode()
    assert version != "0.1"  # (the files' codes; one slot layout since)
    doc = re.search(r"/\* Device view of the resident graph.*?\*/\nint grass_device_view", open(G.INCLUDE).read(), re.S)
    assert f" * {version} on as here" in doc.group(0)
