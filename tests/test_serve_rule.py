"""The server's rule for batches in flight (fg_serve_rule.h), compiled for the host and run
over random orders of launches and completions: while a grid whose CTAs wait on one another
may run, all grids that may run beside it fit on the device together."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

DRIVER = r"""
#include <cstdio>
#include <deque>
#include <random>
#include "fg_serve_rule.h"
struct Batch { bool waits, spread; int ctas, before; };  // before: batches that end before it starts
int main()
{
    std::mt19937 rng(1);
    const int sms = 148;
    long waiting = 0, spread = 0, all = 0;
    for (int slots = 1; slots <= 16; ++slots)
        for (int given = 0; given < 2; ++given) {
            const int cap = sms / slots;
            std::deque<Batch> fly;
            for (int step = 0; step < 20000; ++step) {
                if ((int)fly.size() < slots && rng() % 2) {
                    const bool waits = rng() % 3 == 0;
                    const int grids = 1 + rng() % 3;
                    bool beside = false;
                    for (auto &f : fly) beside = beside || f.waits;
                    const auto m = fg::batch_mode(waits, beside, fly.empty(), given);
                    fly.push_back({waits, m.spread, (m.spread ? grids : 1) * (m.all_sms ? sms : cap),
                                   m.after_spread});
                    waiting += waits; spread += m.spread; all += m.all_sms;
                } else if (!fly.empty()) {
                    fly.pop_front();
                }
                // each waiting batch, with all that may run at the same time
                for (size_t i = 0; i < fly.size(); ++i) {
                    if (!fly[i].waits) continue;
                    int ctas = 0;
                    for (size_t j = 0; j < fly.size(); ++j)
                        if (!(j < i && fly[i].before && fly[j].spread)) ctas += fly[j].ctas;
                    if (ctas > sms) return std::printf("%d slots: %d CTAs beside a waiting grid\n", slots, ctas), 1;
                }
            }
        }
    if (!waiting || !spread || !all) return std::puts("a mode never came up"), 1;
    return 0;
}
"""


def test_waiting_grids_fit_together(tmp_path):
    src, exe = tmp_path / "rule.cpp", tmp_path / "rule"
    src.write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "flashgemm_b200", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout
