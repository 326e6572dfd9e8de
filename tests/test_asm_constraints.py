"""Inline assembly of more than one instruction: an output is written before the last input is read, so it
must not share a register with one (early clobber, "=&")."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "xnyzip_b200", "csrc")


def statements():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            text = f.read()
        for m in re.finditer(r"\basm\b(?:\s+volatile)?\s*\((.*?)\);", text, re.S):
            yield os.path.basename(path), m.group(1)


def test_outputs_of_several_instructions_are_early_clobbers():
    seen = 0
    for path, body in statements():
        strings = re.match(r'\s*(?:"(?:[^"\\]|\\.)*"\s*)+', body).group(0)
        code = "".join(re.findall(r'"((?:[^"\\]|\\.)*)"', strings))
        instructions = [i for i in re.split(r"[;{}]", code) if i.strip() and not i.strip().startswith(".reg")]
        outputs = re.findall(r'"(=[^"]*)"', body[len(strings):])
        if len(instructions) > 1 and outputs:
            seen += 1
            assert all(o.startswith("=&") for o in outputs), (path, body)
    assert seen >= 2
