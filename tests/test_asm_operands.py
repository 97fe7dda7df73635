"""Inline PTX of the kernels: an asm statement of several instructions that writes an output before it has read its last
input has to mark that output as early clobbered ("=&r", "+&r"), or the compiler may keep the output in the register of an
input whose life ends at the statement (carry chains in registers: a sum would be silently wrong)."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "blocksvibe_b200", "csrc")
LITERAL = re.compile(r'"((?:[^"\\]|\\.)*)"')


def statements(text):
    """(line, body) of every asm statement: the text between its parentheses, string literals intact"""
    for m in re.finditer(r"\basm\s+volatile\s*\(|\basm\s*\(", text):
        i, depth = m.end(), 1
        while depth:
            if text[i] == '"':
                i = LITERAL.match(text, i).end()
                continue
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        yield text.count("\n", 0, m.start()) + 1, text[m.end():i - 1]


def sections(body):
    """template, output constraints, input constraints"""
    parts, cur, depth, i = [], "", 0, 0
    while i < len(body):
        c = body[i]
        if c == '"':
            j = LITERAL.match(body, i).end()
            cur += body[i:j]
            i = j
            continue
        depth += {"(": 1, "[": 1, ")": -1, "]": -1}.get(c, 0)
        if c == ":" and depth == 0:
            parts.append(cur)
            cur = ""
        else:
            cur += c
        i += 1
    parts.append(cur)
    template = "".join(LITERAL.findall(parts[0])).replace("\\n", "\n").replace("\\t", "\t")
    lists = [LITERAL.findall(p) for p in parts[1:3]] + [[], []]
    return template, lists[0], lists[1]


def missing_clobbers(body):
    template, outs, ins = sections(body)
    instructions = [x for x in template.split(";") if "%" in x]
    uses = [[int(n) for n in re.findall(r"%(\d+)", x)] for x in instructions]
    dests = []
    for x in instructions:                                   # operands of the first position (one, or a list in braces)
        m = re.match(r"[\s{]*(?:@!?\w+\s+)?[\w.:]+\s+(\{[^}]*\}|[^,]*)", x)
        dests.append([int(n) for n in re.findall(r"%(\d+)", m.group(1))] if m and "[" not in m.group(1) else [])
    last_read = max((i for i, u in enumerate(uses) for n in u if n >= len(outs)), default=-1)
    bad = []
    for n, c in enumerate(outs):
        written = [i for i, d in enumerate(dests) if n in d]
        if written and written[0] < last_read and "&" not in c:
            bad.append(n)
    return bad


def test_checker_sees_a_planted_mistake():
    asm = '"add.cc.u32 %0, %2, %4;\\n\\t" "addc.u32 %1, %3, %5;" : "=r"(x), "=r"(y) : "r"(a), "r"(b), "r"(c), "r"(d)'
    assert missing_clobbers(asm) == [0]
    assert missing_clobbers(asm.replace('"=r"(x)', '"=&r"(x)')) == []
    assert missing_clobbers('"add.u32 %0, %1, %2;" : "=r"(x) : "r"(a), "r"(b)') == []


@pytest.mark.parametrize("name", sorted(os.path.basename(f) for f in glob.glob(os.path.join(CSRC, "*.c*"))))
def test_early_clobbers(name):
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    assert [(line, bad) for line, body in statements(text) if (bad := missing_clobbers(body))] == []
