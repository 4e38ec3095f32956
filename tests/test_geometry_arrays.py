"""Every device array of the mesh (HexGeo) is read by some kernel: an array that
only the upload names holds device memory, and time of every create, for nothing."""

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "gpuwm-hex_b200" / "csrc"


def test_every_mesh_array_is_read():
    struct = re.search(r"struct HexGeo \{(.*?)\n\};", (CSRC / "dycore_geo.cuh").read_text(), re.S).group(1)
    members = re.findall(r"^\s*const \w+\* (\w+);", struct, re.M)
    assert len(members) > 40
    code = "\n".join(re.sub(r"//.*", "", p.read_text()) for p in sorted(CSRC.glob("*.cu*")))
    code = re.sub(r"\bUP\(g\.\w+", "UP(", code)
    unread = [m for m in members if not re.search(rf"\b(?:g|geo)\.{m}\b", code)]
    assert unread == []
