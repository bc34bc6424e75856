"""Sizes that no test graph reaches, checked in the declarations and the host
rules themselves (compiled with the host compiler; no GPU)."""
import os
import subprocess

import pytest

from pgd_gb300 import build as b


def compiled(tmp_path, body):
    """Output of a program whose main is `body`."""
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text('#include <stdio.h>\n#include <type_traits>\n#include "rank_path.h"\n'
                   "int main() {\n%s\nreturn 0;\n}\n" % body)
    r = subprocess.run(["g++", "-std=c++17", "-I" + b.INCLUDE, "-I" + b.CSRC, "-I" + os.path.join(b.CUDA, "include"),
                        "-o", str(exe), str(src)], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    assert r.returncode == 0, r.stdout
    return subprocess.run([str(exe)], stdout=subprocess.PIPE, check=True, text=True).stdout


@pytest.mark.parametrize("field", ["roff", "tw", "eslot", "bend", "bpos"])
def test_slots_are_unsigned(tmp_path, field):
    """A graph of more than 2^30 edges has slots of 2^31 and more: read as signed
    they would index before the arrays."""
    compiled(tmp_path, "static_assert(std::is_same<decltype(pgd_rank_graph::%s), uint32_t *>::value, \"\");" % field)
