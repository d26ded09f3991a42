"""The sample order of training (csrc/epoch_order.h), compiled for the host and driven as
nqb_model_train drives it, with a copy that reads the host array as late as the stream may: at the
wait that ends the epoch.  What the copy sees has to be that epoch's whole permutation."""
import os
import subprocess

import pytest

from conftest import PKG_DIR

DRIVER = r"""
#include <cstdio>
#include <cstdlib>
#include "epoch_order.h"
int main(int, char** a) {
    const uint64_t count = strtoull(a[1], 0, 10), seed = strtoull(a[2], 0, 10);
    const int epochs = atoi(a[3]);
    nqb::EpochOrder order;
    order.start(count, seed);
    for (int ep = 0; ep < epochs; ++ep) {
        const uint32_t* copied_from = order.current();       // the copy is put into the stream
        if (ep + 1 < epochs) order.prepare();                // the host goes on beside the device
        for (uint64_t i = 0; i < count; ++i) printf("%u ", copied_from[i]);  // ... and runs here
        if (ep + 1 < epochs) order.advance();
    }
}
"""


def expected(count, seed, epochs):
    wrap = (1 << 64) - 1
    rng, perm, out = (seed * 0x9E3779B97F4A7C15 + 1) & wrap, list(range(count)), []
    for _ in range(epochs):
        for i in range(count - 1, 0, -1):
            rng = (rng + 0x9E3779B97F4A7C15) & wrap
            z = ((rng ^ (rng >> 30)) * 0xBF58476D1CE4E5B9) & wrap
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & wrap
            j = (z ^ (z >> 31)) % (i + 1)
            perm[i], perm[j] = perm[j], perm[i]
        out += perm
    return out


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    d = tmp_path_factory.mktemp("epoch_order")
    src, exe = os.path.join(d, "driver.cpp"), os.path.join(d, "driver")
    with open(src, "w") as f:
        f.write(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", os.path.join(PKG_DIR, "csrc"), src, "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("count,seed,epochs", [(1, 1, 2), (2, 7, 3), (1000, 1, 1), (1000, 1, 4), (4097, 2**63 + 5, 3)])
def test_a_late_copy_sees_its_own_epoch(driver, count, seed, epochs):
    p = subprocess.run([driver, str(count), str(seed), str(epochs)], check=True, capture_output=True, text=True)
    assert [int(v) for v in p.stdout.split()] == expected(count, seed, epochs)


def test_the_order_outlives_the_stream(nqb):
    # destroyed after the call scope, whose destructor waits for the stream
    with open(os.path.join(PKG_DIR, "csrc", "mlp.cu")) as f:
        body = f.read().split("int nqb_model_train(")[1].split("NQB_ABI_CATCH")[0]
    assert 0 <= body.index("EpochOrder order;") < body.index("CallScope cs(")
