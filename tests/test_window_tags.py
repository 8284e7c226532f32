"""The tags of the messages in windows of steps (window_tags.h), on the CPU: wherever a message is written, the words that lie there from
earlier launches and messages have other tags than its own, both the first word's and the second's."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "genn_b200", "csrc")

HARNESS = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "window_tags.h"
using namespace b200;
int main(int, char **argv)
{
    const unsigned int buffers = windowBuffers(atoi(argv[1])), every = atoi(argv[2]), longest = atoi(argv[3]), launches = atoi(argv[4]);
    if(buffers < (unsigned int)atoi(argv[1])) return 1;
    std::vector<unsigned long long> first(buffers, 0ull);
    std::vector<unsigned int> second(buffers, 0u);
    unsigned int epoch = 0, writtenTo = 0;
    for(unsigned int l = 0; l < launches; l++) {
        bool clear = false;
        epoch = windowNextEpoch(epoch, &clear);
        if(clear) {
            for(unsigned int b = 0; b < writtenTo; b++) { first[b] = 0ull; second[b] = 0u; }
            writtenTo = 0;
        }
        // (a launch has two messages at least)
        const unsigned int messages = l % every ? 2u : longest;
        for(unsigned int m = 0; m < messages; m++) {
            const unsigned int b = m % buffers;
            if(b >= writtenTo) writtenTo = b + 1u;
            if(windowTag(epoch, m) >> 44 || windowShortTag(epoch, m) >> 16) return 2;
            if(first[b] == windowTag(epoch, m)) return 3;
            if(second[b] == windowShortTag(epoch, m)) return 4;
            first[b] = windowTag(epoch, m);
            second[b] = windowShortTag(epoch, m);
        }
    }
    return 0;
}
"""


# sources ahead have 4 buffers, one delay 2 * lag + 2; lags of 127 and 255 would have 256 and 512
@pytest.mark.parametrize("buffers,every,longest,launches", [(4, 256, 4, 5000), (4, 256, 260, 5000), (4, 1, 1000, 3000), (4, 255, 7, 2200000), (16, 256, 300, 20000),
                                                            (256, 256, 700, 20000), (256, 7, 1500, 3000), (512, 256, 1100, 3000), (514, 16, 600, 3000)])
def test_no_word_is_taken_for_one_that_lay_there_before(tmp_path, buffers, every, longest, launches):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no host compiler")
    (tmp_path / "tags.cc").write_text(HARNESS)
    exe = str(tmp_path / "tags")
    subprocess.check_call([gxx, "-std=c++17", "-O2", "-I", CSRC, str(tmp_path / "tags.cc"), "-o", exe])
    assert subprocess.run([exe, str(buffers), str(every), str(longest), str(launches)], timeout=60).returncode == 0
