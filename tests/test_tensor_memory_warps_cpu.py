"""Loads, stores and waits of tensor memory are `.sync.aligned`: the warp's lanes have to come to them together. Lanes that have
parted (a store that some of them leave out, one more trip through a loop) are brought together by the helpers themselves."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "edge-infer_b200" / "csrc"
COLLECTIVE = re.compile(r'"tcgen05\.(?:ld|st|wait::ld|wait::st)\.sync\.aligned')


def test_helpers_bring_the_warp_together():
    found = 0
    for path in sorted(CSRC.glob("*.cu*")):
        text = path.read_text()
        for match in COLLECTIVE.finditer(text):
            body = text[text.rindex("__device__", 0, match.start()):match.start()]
            assert "__syncwarp();" in body, f"{path.name}: {text[match.start():match.start() + 40]}"
            found += 1
    assert found >= 8
