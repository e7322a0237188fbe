"""CPU checks of rules that the kernels' sources have to keep and that no run can show."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "spargeattn_b200", "csrc")


def _waiting_kernels():
    """(name, parameters, body) of every kernel that may run beside the one before it."""
    found = []
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
        for m in re.finditer(r"__global__.*?(\w+_kernel)\((.*?)\)\s*\{\n(.*?)\n\}\n", text, flags=re.S):
            if "pdl_wait" in m.group(3):
                found.append(m.groups())
    return found


def test_kernels_that_wait_for_the_one_before_do_not_claim_constant_inputs():
    kernels = _waiting_kernels()
    assert {k[0] for k in kernels} >= {"prep_combine_kernel", "prep_second_kernel", "select_kernel", "mask_to_lut_kernel", "row_order_kernel", "attn_kernel"}
    for name, parameters, _ in kernels:
        for parameter in parameters.split(","):
            assert not ("const" in parameter and "__restrict__" in parameter), (name, parameter)


def _unconditional_wait(body):
    """Where the wait stands that every block comes to (it may have waited in a branch before), or the end of the body."""
    depth = 0
    for m in re.finditer(r"[{}]|pdl_wait\(\);", body):
        depth += {"{": 1, "}": -1}.get(m.group(), 0)
        if depth == 0 and m.group() == "pdl_wait();":
            return m.start()
    return len(body)


def test_no_block_returns_before_it_has_waited():
    """A return in front of the wait that all blocks come to has a wait of its own, in the statement before it."""
    for name, _, body in _waiting_kernels():
        head = body[:_unconditional_wait(body)]
        for m in re.finditer(r"\breturn;", head):
            assert re.search(r"pdl_wait\(\);\s*$", head[:m.start()]), name


def test_heads_are_grouped_evenly(tmp_path):
    """Groups of heads follow one another, cover all heads, differ by one head at most, and a head finds its own."""
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    src = tmp_path / "groups.cpp"
    src.write_text('''
#include <initializer_list>
#include "row_groups.cuh"
int main() {
  using namespace sparge;
  for (int heads : {1, 2, 3, 13, 16, 24, 25, 26, 60, 997, 65535})
    for (int groups = 1; groups <= heads; groups += heads < 1000 || groups < 40 || groups > heads - 40 ? 1 : 611) {
      int next = 0;
      for (int g = 0; g < groups; g++) {
        const HeadGroup h = head_group(g, heads, groups);
        if (h.first != next || h.heads < heads / groups || h.heads > (heads + groups - 1) / groups) return 1;
        if (group_of_head(h.first, heads, groups) != g || group_of_head(h.first + h.heads - 1, heads, groups) != g) return 2;
        next = h.first + h.heads;
      }
      if (next != heads) return 3;
    }
  return 0;
}
''')
    subprocess.run([gxx, "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(tmp_path / "groups")], check=True)
    assert subprocess.run([str(tmp_path / "groups")]).returncode == 0


def test_any_step_word_names_a_block_of_the_row(tmp_path):
    """The softmax warps go on after an expired wait, on whatever the word in shared memory then holds."""
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    src = tmp_path / "words.cpp"
    src.write_text('''
#include <initializer_list>
#include "step_word.cuh"
int main() {
  using namespace sparge;
  for (int nk : {1, 2, 63, 1861, 65535}) {
    for (unsigned w = 0; w < 1u << 16; w++)
      for (unsigned hi : {0u, 0x8000u, 0x7fffu, 0xffffu, 0x1234u}) {
        const int j = step_block((int)(hi << 16 | w), nk);
        if (j < 0 || j >= nk) return 1;
      }
    for (int j = 0; j < nk; j++)
      for (bool m : {false, true})
        if (step_block(step_word(j, m), nk) != j || step_masked(step_word(j, m)) != m) return 2;
  }
  return 0;
}
''')
    subprocess.run([gxx, "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(tmp_path / "words")], check=True)
    assert subprocess.run([str(tmp_path / "words")]).returncode == 0
    # every load that takes the word is through step_block; step_index feeds the key masks
    text = open(os.path.join(CSRC, "attn_sm100.cu")).read()
    assert re.findall(r"(\S+) step_index\(word\) \* 64;", text) == ["="] and text.count("step_index(") == 1
    assert text.count("(size_t)step_block(word, nk)") == text.count("step_block(") == 1
