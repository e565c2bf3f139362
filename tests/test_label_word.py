"""The word of a label search (csrc/gsofa_label.h), on the CPU: every order in
which an expansion and two improvements of one id can take their single atomic
operations.  No improvement may be lost: whatever the order, the expansions
that follow from the queue read the smallest label in the end, and the id is
never on the queue twice."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "gsofa_label.h"
using namespace gsofa;

struct State {
    int word, listed, last_read, expanding;  // listed: entries on the queues
    int label[2], seen[2], step[2];
};

static long long ends = 0;
static void fail(const char* why) { std::printf("%s\n", why); std::exit(1); }

static void expand(State& s) {  // one operation: mark idle, read the label
    s.last_read = label_of_word(s.word);
    s.word |= kLabelIdle;
    s.listed--;
}

static void improve(State& s, int i) {
    if (s.step[i] == 0) {  // look
        s.seen[i] = s.word;
        s.step[i] = s.label[i] < label_of_word(s.seen[i]) ? 1 : 2;
        return;
    }
    const int w = label_queued(s.label[i]), before = s.word;  // one operation: the minimum
    if (w < s.word) s.word = w;
    if (label_queues(before, w)) s.listed++;
    s.step[i] = 2;
}

static void walk(State s) {
    if (s.listed > 1) fail("listed twice");
    bool more = false;
    if (s.listed == 1) {
        State t = s;
        expand(t);
        walk(t);
        more = true;
    }
    for (int i = 0; i < 2; i++) {
        if (s.step[i] == 2) continue;
        State t = s;
        improve(t, i);
        walk(t);
        more = true;
    }
    if (more) return;
    ends++;
    if (s.last_read != label_of_word(s.word)) fail("an improvement was lost");
    if (!(s.word & kLabelIdle)) fail("queued and not listed");
}

int main() {
    for (int first = 0; first < 4; first++)  // the label before; 3: none yet
        for (int a = 0; a < 3; a++)
            for (int b = 0; b < 3; b++) {
                State s{};
                s.last_read = -1;
                if (first == 3) s.word = kNoLabelWord;
                else s.word = label_queued(first), s.listed = 1;
                s.label[0] = a;
                s.label[1] = b;
                walk(s);
            }
    static_assert(label_of_word(kNoLabelWord) >= (1 << 30) - 1, "above every id");
    std::printf("%lld\n", ends);
    return 0;
}
"""


def test_no_order_loses_an_improvement(tmp_path):
    src, exe = tmp_path / "label.cpp", tmp_path / "label"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I",
                    os.path.join(ROOT, "gsofatpds_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    assert int(out.stdout) > 100
