"""Rules of the kernels' dispatch that the code states once, or that hold only in bounds the host has to check: on the sources,
and on the host functions themselves in a program of their own."""
import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parent.parent / "c0ven_b200" / "csrc"


def function(path, name):
    """The definition of the function `name`, comments left out."""
    text = re.sub(r"//[^\n]*", "", (CSRC / path).read_text())
    at = re.search(r"\b" + name + r"\([^;{]*\{", text)
    depth = 0
    for i in range(at.end() - 1, len(text)):
        depth += (text[i] == "{") - (text[i] == "}")
        if depth == 0:
            return text[at.start():i + 1]
    raise ValueError(name)


def test_the_specialised_row_lengths_are_listed_once():
    """The rule for groups of two rows asks whether the integer-dot kernels are specialised for a length: by the list that their
    dispatch instantiates them from, not by one of its own."""
    rule, dispatch = function("moe_layer.cu", "groups_take_mma"), function("expert_rows_inst.cuh", "launch_shape")
    assert "rows_specialised(" in rule and "rows_specialised(" in dispatch
    for text in (rule, dispatch):
        assert not re.search(r"\b(2048|512|256)\b", text)
