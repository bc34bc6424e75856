"""Sizes that no test graph reaches, checked in the declarations and the host
rules themselves (compiled with the host compiler; no GPU)."""
import os
import subprocess

import pytest

from pgd_gb300 import build as b


def compiled(tmp_path, body):
    """Output of a program whose main is `body`."""
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text('#include <stdio.h>\n#include <type_traits>\n#include "rank_path.h"\n#include "size_rules.h"\n'
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


@pytest.mark.parametrize("max_id", [-1, 0, 1, 6, 7, 2 ** 20 - 1, 2 ** 30, 2 ** 31 - 2, 2 ** 31 - 1])
def test_packed_words_hold_every_id(tmp_path, max_id):
    """A word of row and column takes every id up to the largest and the row behind
    them, in at most 64 bits."""
    out = compiled(tmp_path, 'printf("%%d", pgd_id_bits((int32_t)%dll));' % max_id)
    bits = int(out)
    assert max_id + 1 < 2 ** bits and bits <= 32 and bits == max(1, (max_id + 1).bit_length())


@pytest.mark.parametrize("n,entries", [(2 ** 31 - 2 ** 16, 2), (2 ** 31 - 16385, 2 ** 20), (2 ** 31 - 1, 2), (2 ** 31, 0),
                                       (2 ** 31, 2 ** 32 - 2)])
def test_core_kernels_that_count_in_32_bits_take_no_such_graph(tmp_path, n, entries):
    """Few edges on large ids: the cluster's loops over vertices would pass 2^31."""
    out = compiled(tmp_path, 'printf("%%d %%d", pgd_core_light(%dll, %dll), pgd_core_narrow(%dll, %dll, 64, 0, 0));'
                   % (n, entries, n, entries))
    assert out == "0 0"


def test_core_choice_follows_the_measured_sides(tmp_path):
    """Light graphs by the cluster, wide ones by the device until their steps are narrow."""
    light = [(1, 0), (65473, 1818884), (262144, 5242608), (4194304, 999926), (1048576, 4194282)]
    heavy = [(262144, 6291128), (16777216, 999926), (4194305, 8388608), (1048576, 52427448), (100, 2 ** 32 - 2)]
    body = "".join('printf("%%d", pgd_core_light(%dll, %dll));' % x for x in light + heavy)
    # steps of a path (two vertices leave), and of a random graph (every vertex scanned again and again)
    body += 'printf("%d%d", pgd_core_narrow(4000000, 8000000, 64, 0, 128), ' \
            'pgd_core_narrow(1048576, 52427448, 64, 20000000, 1000));'
    assert compiled(tmp_path, body) == "1" * len(light) + "0" * len(heavy) + "10"


# n, p, share, edge by edge: clearly faster on its side in the times beside the rule
SAMPLES = [(1000, 0.5, 1 / 2048, 1), (1000, 0.5, 1 / 512, 1), (1000, 0.5, 1 / 64, 0), (1000, 0.9, 1 / 16, 1),
           (1000, 0.9, 1 / 4, 0), (2000, 0.5, 1 / 256, 1), (2000, 0.5, 1 / 8, 0), (3000, 0.5, 1 / 16, 1),
           (5000, 0.2, 1 / 2048, 1), (5000, 0.2, 1 / 512, 0), (250, 0.9, 1 / 2048, 0), (1000, 0.25, 1 / 2048, 0),
           (3000, 0.1, 1 / 2048, 0), (1 << 20, 3e-5, 1 / 2000, 0), (1 << 20, 3e-5, 1 / 10000, 1), (3000, 0.9, 1, 0),
           (20000, 1.0, 1, 0), (3, 1.0, 1, 0)]


def test_samples_take_the_faster_path(tmp_path):
    body = ""
    for n, p, share, _ in SAMPLES:
        m = int(p * n * (n - 1) / 2)
        body += 'printf("%%d", pgd_sample_edgewise(%dll, %dll, %dll));' % (n, m, max(1, int(share * m)))
    body += 'printf("%d%d", pgd_sample_edgewise(5, 0, 0), pgd_sample_edgewise(0, 0, 0));'
    assert compiled(tmp_path, body) == "".join(str(s[3]) for s in SAMPLES) + "00"
