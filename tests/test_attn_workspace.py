"""-m "not gpu": where one-token attention's split partials lie in the caller's workspace (csrc/attn_workspace.h), over all head counts and
numbers of multiprocessors that lead to odd products of KV heads, splits and query heads: the 16-byte reads of the merge are aligned, nothing overlaps, all
lies inside the bytes that yalm_attn_workspace_bytes states."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "attn_workspace.h"
#include <algorithm>
#include <cstdio>
int main() {
	long n = 0;
	for (int sms = 1; sms <= 200; ++sms)
		for (int n_kv = 1; n_kv <= 130; ++n_kv)
			for (int g = 1; g <= 8; g *= 2)
				for (int hd = 16; hd <= 128; hd *= 2)
					for (uintptr_t at = 4096; at < 4096 + 16; at += 4) {
						const int S = std::max(1, std::min(512, 2 * sms / n_kv));
						const yalm::AttnWorkspace w = yalm::attn_workspace(at, n_kv, S, g, hd);
						const size_t rows = (size_t)n_kv * S * g;
						const bool ok = (at + w.acc) % 16 == 0 && (at + w.ml) % 4 == 0 && w.acc >= 4 * (size_t)n_kv && (at % 16 || w.acc >= 256) &&
						                w.ml >= w.acc + rows * hd * 4 && w.ml + rows * 8 <= w.bytes && w.bytes == rows * (hd + 2) * 4 + 4 * (size_t)n_kv + 256;
						if (!ok) return std::printf("sms %d kv heads %d group %d head size %d at %zu\n", sms, n_kv, g, hd, (size_t)at), 1;
						++n;
					}
	std::printf("%ld\n", n);
	return 0;
}
"""


def test_partials_are_aligned_and_inside(tmp_path):
    src, exe = tmp_path / "ws.cpp", tmp_path / "ws"
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "yalm_b200", "csrc"), str(src), "-o", str(exe)])
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
    assert int(r.stdout) == 200 * 130 * 4 * 4 * 4
