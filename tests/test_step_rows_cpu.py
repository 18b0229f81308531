"""Rows of a step of the config.json families, for every token_chunk_size: no launch covers more rows than the buffers hold, and the walk that sizes the
projections' workspace visits every row count a launch can have.  The arithmetic itself (csrc/kx_rows.cuh is plain C++), compiled here."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ai00_server_b200", "csrc")

MAIN = r"""
#include <cstdio>
#include <set>
#include "kx_rows.cuh"
using namespace b200;
int main() {
    int bad = 0;
    for (int chunk : {1 << 30, 65536, 4096, 2049}) bad += kx_max_rows(chunk, false) != KX_MAX_STEP;
    for (int chunk = 1; chunk <= 2048; ++chunk)
        for (bool exact : {false, true}) {
            const int rows = kx_max_rows(chunk, exact), out = std::min(rows, KX_MAX_OUT_ROWS), portion = kx_portion(chunk);
            std::set<int> walked;
            for (int r = rows; r > 16; r = kx_bucket_below(r)) walked.insert(r);
            const int step = kx_step_tokens(chunk, exact), cap = std::min(chunk, portion);      // tokens of a step, of a portion
            bool ok = rows >= portion && out >= cap && rows >= step && step >= cap && step == (exact ? cap : std::min(16 * chunk, 2048));
            for (int n = 1; n <= rows; ++n) ok = ok && kx_bucket(n) >= n && kx_bucket(n) <= rows && (kx_bucket(n) <= 16 || walked.count(kx_bucket(n)));
            for (int n = 1; n <= out; ++n) ok = ok && kx_bucket(n) <= out;
            if (!ok && bad++ < 20) printf("chunk %d exact %d: buffers of %d rows, a full step's launches have %d, %d logits rows' %d\n", chunk, exact, rows, kx_bucket(rows), out, kx_bucket(out));
        }
    return bad ? 1 : 0;
}
"""


def test_no_step_has_more_rows_than_its_buffers(tmp_path):
    src, exe = tmp_path / "rows.cpp", tmp_path / "rows"
    src.write_text(MAIN)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-x", "c++", "-I", CSRC, str(src), "-o", str(exe)])
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
