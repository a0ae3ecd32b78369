"""Carry chains hand the carry flag from one asm statement to the next, and the compiler
keeps only volatile statements in order among themselves: every statement that reads or
writes the flag has to be volatile."""
from __future__ import annotations

import glob
import os
import re

from conftest import ROOT


def statements(text):
    """(qualifier, body) of every asm statement, the body up to its closing bracket."""
    for m in re.finditer(r"\basm\s*(volatile)?\s*\(", text):
        depth, i, quoted = 1, m.end(), False
        while depth:
            c = text[i]
            if c == '"':
                quoted = not quoted
            elif not quoted:
                depth += (c == "(") - (c == ")")
            i += 1
        yield m.group(1), text[m.end():i]


def test_flag_users_are_volatile():
    seen = 0
    for path in sorted(glob.glob(os.path.join(ROOT, "ppopp26-artifact_gb300", "csrc", "*.cu*"))):
        with open(path) as f:
            for qualifier, body in statements(f.read()):
                # PP_ASM macros take the instruction's name as an argument
                if re.search(r"\.cc\b|\b(addc|subc|madc)\b", body) or re.match(r"op\b", body.strip()):
                    seen += 1
                    assert qualifier == "volatile", (os.path.basename(path), body[:60])
    assert seen >= 3
