"""Launch sizes of the tiled kernels: computed without wrapping, and checked by
the dispatch against the smallest tile of the variant it picked before anything
is launched.  (A call that reaches the limit needs more memory than a GPU has.)"""
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "yell_gb300", "csrc")


def test_launch_sizes(tmp_path):
    exe = tmp_path / "launch_size_test"
    r = subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CSRC}", f"{ROOT}/tests/cpp/launch_size_test.cpp", "-o",
                        str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "OK", r.stdout


def test_the_dispatch_checks_before_it_launches():
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "ntt_dispatch.cu")).read())
    for name, launch in (("launch_ntt", "v.ntt("), ("launch_polymul", "v->polymul(")):
        body = text[text.index(f"cudaError_t {name}("):]
        body = body[:body.index("\n}")]
        assert 0 < body.index("one_launch(") < body.index(launch), name
