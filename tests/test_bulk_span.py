"""The conjugate gradient's bulk copies stay inside the value array (csrc/pfg_bulk_span.h,
compiled here for the host)."""
import os
import shutil
import subprocess

import pytest

from conftest import REPO

PROGRAM = r"""
#include "pfg_bulk_span.h"
#include <cstdio>
#include <vector>
int main()
{
	for (int odd = 0; odd < 2; ++odd)
		for (int n = 1; n <= 40; ++n)
			for (int v0 = 0; v0 < n; ++v0)
				for (int nv = 0; v0 + nv <= n; ++nv)
				{
					const int at = (odd + v0) & 1; // the chunk's first value, modulo a 16-byte unit
					const pfg::BulkSpan s = pfg::bulk_span(v0, nv, n, at);
					std::vector<char> got(n + 1, 0);
					bool bad = s.end < s.begin || ((s.end - s.begin) & 1);
					if (s.end > s.begin)
						bad = bad || v0 + s.begin < 0 || v0 + s.end > n || ((at + s.begin) & 1) || at + s.begin < 0;
					for (int k = s.begin; k < s.end && !bad; ++k) got[v0 + k] = 1;
					if (s.lo) got[v0] = 1;
					if (s.hi) got[v0 + nv - 1] = 1;
					for (int k = 0; k < nv; ++k) bad = bad || !got[v0 + k];
					bad = bad || (nv == 0 && (s.end > s.begin || s.lo || s.hi));
					if (bad) return std::printf("odd %d n %d v0 %d nv %d: [%d, %d)\n", odd, n, v0, nv, s.begin, s.end), 1;
				}
	return 0;
}
"""


def test_every_copy_starts_on_16_bytes_inside_the_array(tmp_path):
    """Every chunk of every array of up to 40 values, at both alignments: the copy is whole
    16-byte units within the array, and with the single loads it covers the chunk."""
    cxx = shutil.which(os.environ.get("CXX", "g++"))
    if cxx is None:
        pytest.skip("no C++ compiler")
    src = tmp_path / "span.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "span"
    subprocess.check_call([cxx, "-std=c++17", "-I", os.path.join(REPO, "polyfem_b200", "csrc"), str(src), "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
