"""Dynamic shared memory is declared with the alignment of the widest vector that is
read from it: an array of scalars is aligned to the scalar only, and 8- or 16-byte
accesses to it then depend on what the kernel's other arrays happen to be."""

import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parents[1] / "beamax_b200" / "csrc"
SIZE = {"char": 1, "uint8_t": 1, "float": 4, "int": 4, "double": 8, "float2": 8, "int2": 8, "float4": 16, "int4": 16, "double2": 16}


def test_dynamic_shared_arrays_are_aligned_for_their_vectors():
    seen = 0
    for f in sorted(CSRC.glob("*.cu*")):
        text = f.read_text()
        for m in re.finditer(r"extern\s+__shared__\s+(?:__align__\((\d+)\)\s+)?(?:unsigned\s+)?(\w+)\s+(\w+)\[\]", text):
            have = max(int(m.group(1) or 0), SIZE[m.group(2)])
            # the vectors the file casts this array to, directly or with an offset
            need = [SIZE[t] for t in re.findall(r"reinterpret_cast<(?:typename\s+)?(\w+)\s*\*>\(\s*" + m.group(3) + r"\b", text)
                    if t in SIZE]
            # (a dependent vector type counts as the widest)
            if re.search(r"reinterpret_cast<typename [^;]*\*>\(\s*" + m.group(3) + r"\b", text):
                need.append(16)
            seen += 1
            assert have >= max(need, default=1), (f.name, m.group(3), have, need)
    assert seen >= 4
