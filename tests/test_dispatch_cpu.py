"""Rules of the kernels' dispatch that the code states once, or that hold only in bounds the host has to check: on the sources,
and on the host functions themselves in a program of their own."""
import pathlib
import re
import subprocess

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


def test_items_are_divided_exactly_up_to_what_the_host_admits(tmp_path):
    """The tile kernels divide an item's number by the items a tile has with a multiply: for every layer size at the largest
    count of tiles that the launch admits, around every multiple; and one tile more is refused, in the launch."""
    program = r"""
#include <cstdio>
#include <initializer_list>
#include "formats.h"
using namespace moe;
int main() {
  for (uint32_t n = 1; n <= 64; n++) {
    uint64_t tiles = ((1ull << 32) - 1) / n / n;
    while (items_divide(tiles + 1, n)) tiles++;
    while (tiles && !items_divide(tiles, n)) tiles--;
    if (!tiles || items_divide(tiles + 1, n) || items_divide(1ull << 32, n)) return 1;
    const uint64_t items = tiles * n;
    const uint32_t magic = item_magic(n);
    auto quotient = [&](uint64_t i) { return n > 1 ? (i * magic) >> 32 : i; };
    for (uint64_t t = 0; t < tiles; t += t < 4096 || t + 4096 > tiles ? 1 : 997)
      for (uint64_t i : {t * n, t * n + n / 2, t * n + n - 1})
        if (i >= items || quotient(i) != t) return 2;
  }
  puts("exact");
}
"""
    (tmp_path / "divide.cpp").write_text(program)
    subprocess.run(["g++", "-std=c++17", "-O2", "-I" + str(CSRC), str(tmp_path / "divide.cpp"), "-o", str(tmp_path / "divide")], check=True)
    assert subprocess.run([str(tmp_path / "divide")], capture_output=True, text=True).stdout == "exact\n"
    assert "!items_divide(max_tiles," in function("expert_tiles_inst.cuh", "launch_expert_tiles")
    assert "item_magic(" in (CSRC / "expert_tiles.cuh").read_text()


def test_what_a_launch_keeps_is_kept_for_one_kernel():
    """What a launch asks the device once and keeps (an attribute set, clusters that fit) lies in a static word, which has to be one
    a kernel: a helper that is a template on the kernel's type alone has one for all kernels of that signature."""
    statics = 0
    for path in sorted(CSRC.glob("*.cu*")) + sorted(CSRC.glob("*.h")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"static std::atomic<[^;]*;", text):
            statics += 1
            templates = [t for t in re.finditer(r"^template <([^\n]*)>$", text[:m.start()], re.M)]
            start = [f for f in re.finditer(r"^(?!template|namespace|//)[\w:]+ [^;\n]*\([^;]*?\{$", text[:m.start()], re.M)][-1]
            own = [t.group(1) for t in templates if text[t.end():start.start()].strip() == ""]
            assert not own or not re.fullmatch(r"(class|typename) \w+", own[0]), (path.name, start.group(0))
    assert statics >= 7  # the pattern still finds them
