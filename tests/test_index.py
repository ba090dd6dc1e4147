"""CPU check of the index arithmetic of the density pass's lists and chunks
(upbd_index.h, the code the kernels run) up to the largest scene the library
accepts: list rows past 2^32 entries, slots past 2^28."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]

SRC = r"""
#include <cstdio>
#include <initializer_list>
#include "upbd_index.h"
using namespace upbd;
int main() {
  const uint32_t ns[] = {1u, 73536u, 38347922u, 38347923u, 159072863u, (1u << 28) - 1u, 1u << 28, (1u << 28) + 1u, 1u << 29};
  for (uint32_t n : ns) {
    if (n > MAX_PARTICLES) return 1;
    for (uint32_t row : {0u, 1u, NL - 1u, NL, GLF * NL - 1u})
      printf("r %u %u %llu\n", n, row, (unsigned long long)list_row_bytes(row, n));
    // a place and a slot of one bucket of b particles at either end of the table
    for (uint32_t b : {1u, 2u, 9u, 100001u})
      for (uint32_t at : {0u, n - (b < n ? b : n)})
        for (uint32_t size = 0; size <= CHUNK; size++)
          for (int swap = 0; swap < 2; swap++) {
            const uint32_t lo = at, hi = at + (b < n ? b : n) - 1u;
            const uint32_t place = swap ? hi : lo, slot = swap ? lo : hi, w = chunk_word(place, slot, size);
            if (chunk_word_size(w) != size || chunk_word_slot(place, w) != slot) return 2;
          }
  }
  // the bucket's own limit
  const uint32_t far = (1u << 27) - 1u;
  if (chunk_word_slot(far, chunk_word(far, 0u, CHUNK)) != 0u || chunk_word_slot(0u, chunk_word(0u, far, 1u)) != far) return 3;
  printf("max %lld\n", (long long)MAX_PARTICLES);
  return 0;
}
"""


def test_list_rows_and_chunk_words_at_every_accepted_size(tmp_path):
    (tmp_path / "i.cpp").write_text(SRC)
    exe = tmp_path / "i"
    subprocess.run(["g++", "-std=c++17", "-I", str(ROOT / "fluidphysics_b200" / "csrc"), str(tmp_path / "i.cpp"), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.returncode
    rows = [r.split() for r in out.stdout.splitlines()]
    assert rows[-1] == ["max", str(1 << 29)]
    for _, n, row, got in (r for r in rows if r[0] == "r"):
        assert int(got) == 4 * int(n) * int(row)


def test_the_kernels_index_their_lists_through_it():
    """No product of a list row and the slot count is left in 32 bits."""
    text = (ROOT / "fluidphysics_b200" / "csrc" / "upbd_passes.cuh").read_text()
    assert "* NS]" not in text and "CHUNK_SLOT" not in text
    assert text.count("list_entry(") >= 6
