"""CPU test of the inline PTX in csrc: what a compiler may assume of an asm statement's operands holds for it."""
import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "strixite_b200" / "csrc"


def asm_statements(text):
    """(line, inside of the parentheses) of every asm statement."""
    for m in re.finditer(r"\basm\s*(?:volatile)?\s*\(", text):
        i, depth, quoted = m.end(), 1, False
        while depth:
            c = text[i]
            if quoted:
                i += c == "\\"
                quoted = c != '"'
            elif c == '"':
                quoted = True
            else:
                depth += (c == "(") - (c == ")")
            i += 1
        yield text.count("\n", 0, m.start()) + 1, text[m.end():i - 1]


def parse(body):
    """(instructions, constraints of the outputs, count of the inputs); braces and declarations stay part of their instruction."""
    strings = r'"(?:[^"\\]|\\.)*"'
    code = re.match(rf"\s*((?:{strings}\s*)+)", body)
    instructions = "".join(s[1:-1] for s in re.findall(strings, code.group(1))).replace("\\n", " ").replace("\\t", " ").split(";")
    sections = [""]
    for part in re.findall(rf"{strings}|:|[^\":]+", body[code.end():].replace("::", ": :")):
        if part == ":":
            sections.append("")
        else:
            sections[-1] += part
    operands = [re.findall(r'"([^"]*)"\s*\(', s) for s in sections]
    return instructions, operands[1] if len(operands) > 1 else [], len(operands[2]) if len(operands) > 2 else 0


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cu*")), ids=lambda p: p.name)
def test_outputs_written_before_the_last_input_is_read_are_early_clobbers(path):
    """An output without '&' may share its register with an input; an instruction that writes it must not come before one that reads that input."""
    for line, body in asm_statements(path.read_text()):
        instructions, outputs, n_in = parse(body)
        uses = [{int(k) for k in re.findall(r"%(\d+)", s)} for s in instructions]
        last_input = max((i for i, u in enumerate(uses) if any(len(outputs) <= k < len(outputs) + n_in for k in u)), default=-1)
        for k, constraint in enumerate(outputs):
            first = min((i for i, u in enumerate(uses) if k in u), default=len(uses))
            assert "&" in constraint or first >= last_input, f"{path.name}:{line}: output %{k} ('{constraint}') is written before the last input is read"
