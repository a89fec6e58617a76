"""The rule by which a grid's latitude pairs take the two-degree recurrence
(charm_b200/csrc/lat_pairs.h), compiled for the host: it reads the array it is
given and nothing before or behind it (the array stands alone between two pages
that cannot be read), and splits the pairs as its comment says."""
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "charm_b200", "csrc")

MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <sys/mman.h>
#include <unistd.h>
#include <vector>
#include "lat_pairs.h"

// the array at the very start (0) or end (1) of readable memory
static double *place(const std::vector<double> &v, int end)
{
    const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    const size_t len = (v.size() * 8 + page - 1) / page * page;
    char *m = (char *)mmap(nullptr, len + 2 * page, PROT_NONE,
                           MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    mprotect(m + page, len, PROT_READ | PROT_WRITE);
    char *at = m + page + (end ? len - v.size() * 8 : 0);
    std::memcpy(at, v.data(), v.size() * 8);
    return (double *)at;
}

int main()
{
    int np;
    while (std::scanf("%d", &np) == 1)
    {
        std::vector<double> v(np);
        for (double &x : v)
            if (std::scanf("%lf", &x) != 1)
                return 1;
        int n2[2], polar[2];
        for (int e = 0; e < 2; e++)
        {
            polar[e] = -1;
            n2[e] = cb::two_pairs(place(v, e), np, &polar[e]);
        }
        if (n2[0] != n2[1])
            return 2;
        std::printf("%d %d\n", n2[0], polar[0]);
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def two_pairs(tmp_path_factory):
    cxx = next((c for c in ("/usr/bin/g++", "g++") if shutil.which(c)), None)
    if cxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("lat_pairs")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", CSRC, "main.cpp", "-o",
                    "main"], cwd=d, check=True)

    def run(*lats):
        text = "".join("%d %s\n" % (len(v), " ".join("%.17g" % x for x in v))
                       for v in lats)
        r = subprocess.run([str(d / "main")], input=text, capture_output=True,
                           text=True)
        assert r.returncode == 0, r.returncode
        return [tuple(map(int, l.split())) for l in r.stdout.splitlines()]
    return run


@pytest.mark.parametrize("np_", [1, 31, 32, 33, 64, 96, 512])
def test_every_pair_at_the_equator(two_pairs, np_):
    """No pair outside the equatorial band: none taken, whole groups or not
    (the rest below a whole group may be where it lies outside 0.8 of it)."""
    a = np.linspace(0.038, 0.001, np_)
    assert two_pairs(a, -a, a * 0.0) == [(0, 0)] * 3
    b = np.linspace(0.0499, 0.001, np_)
    (n2, polar), = two_pairs(b)
    assert n2 in (0, np_ % 32) and polar == 0


def test_whole_groups_beside_the_equator(two_pairs):
    near, far = np.linspace(0.0499, 0.0001, 100), np.linspace(1.5, 0.06, 70)
    (n2, polar), = two_pairs(np.concatenate([far, near]))
    # 170 pairs: 96 of the 100 stay in whole groups, four join the others
    assert n2 == 74
    assert polar == 32 * (np.count_nonzero(far >= np.pi / 6) // 32)
    # not where that would leave pairs within 0.8 of the band to the others
    near = np.linspace(0.0399, 0.0001, 100)
    assert two_pairs(np.concatenate([far, near]))[0][0] == 70


def test_orders_that_are_not_taken(two_pairs):
    up = np.linspace(0.1, 1.5, 64)
    one = np.linspace(1.5, 0.1, 64)
    one[40] = one[38]
    bad = np.linspace(1.5, 0.1, 64)
    bad[10] = np.nan
    first = np.linspace(1.5, 0.1, 64)
    first[0] = np.nan
    assert [t[0] for t in two_pairs(up, one, bad, first)] == [0, 0, 0, 0]
    assert two_pairs(np.linspace(1.5, 0.1, 64), np.full(5, 0.3)) == [
        (64, 32), (5, 0)]
