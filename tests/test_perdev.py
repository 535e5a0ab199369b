"""Per-device scratch state (csrc/dn_perdev.h): calls on different devices do not wait for one
another, calls on one device do, and a device's slot stays the same object."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "denise-black-edition_b200", "csrc")

PROGRAM = r"""
#include <thread>
#include "dn_perdev.h"
int main()
{
    PerDevice<int> p;
    auto *a = &p.at(0);
    std::lock_guard<std::mutex> lk(a->mu);   // a call on device 0 under way
    bool other = false, same = true;
    std::thread([&] { auto &s = p.at(1); other = s.mu.try_lock(); if (other) s.mu.unlock(); }).join();
    std::thread([&] { same = p.at(0).mu.try_lock(); }).join();
    for (int d = 2; d < 64; d++) p.at(d).value = d;
    return other && !same && a == &p.at(0) && p.at(1).value == 0 && p.at(63).value == 63 ? 0 : 1;
}
"""


def test_one_lock_per_device(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-pthread", "-I", CSRC, str(src), "-o", str(exe)])
    subprocess.check_call([str(exe)], timeout=20)


def test_gradient_readback_uses_it():
    """dn_model_get_gradient holds its own device's lock and no other."""
    text = open(os.path.join(CSRC, "dn_engine.cu")).read()
    body = text[text.index('extern "C" int dn_model_get_gradient'):]
    body = body[:body.index("\n}\n")]
    assert body.count("lock_guard") == 1 and "g_grad_scratch.at(m->device)" in body
