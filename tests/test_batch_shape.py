"""The cluster size of a batched multigrid launch (csrc/batch_shape.h, built for the host) on batches timed
on a B200 with 16, 8 and 4 CTAs per cluster: at most 5 % above the size their number alone would take, and
at most 5 % above the fastest where one system is more than seven times the others."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cicy_geom_b200", "csrc")
MAIN = """
#include <cstdio>
#include <cstdlib>
#include "batch_shape.h"
int main(int argc, char** argv) {
    std::vector<int> rows;
    for (int i = 4; i < argc; i++) rows.push_back(atoi(argv[i]));
    const int resident[3] = {atoi(argv[1]), atoi(argv[2]), atoi(argv[3])};
    printf("%d", cicy::mg_batch_shape(rows, resident));
}
"""
# rows of the systems, ms with 16, 8 and 4 CTAs per cluster
MEASURED = [([2344], (0.729, 0.739, 0.793)), ([120445], (8.17, 12.32, 20.8)), ([2344] * 8, (1.387, 1.191, 1.284)),
            ([2344] * 24, (3.186, 1.905, 1.276)), ([2344] * 24 + [18073], (3.980, 3.917, 5.665)),
            ([2344] * 20 + [58149], (7.243, 10.552, 17.439)), ([2344] * 7 + [120445] * 3, (9.798, 14.482, 23.702)),
            ([7140] * 8, (2.672, 2.003, 2.700)), ([7140] * 24, (5.881, 3.574, 2.681)), ([7140] * 8 + [18073], (3.088, 3.952, 5.716)),
            ([7140] * 20 + [18073], (5.419, 3.954, 5.715)), ([7140] * 24 + [58149], (7.302, 10.530, 17.418)),
            ([2344] * 24 + [7140] * 24 + [18073], (8.494, 4.602, 5.765)), ([2344] * 24 + [7140] * 24 + [58149], (9.467, 10.654, 17.584)),
            ([2344] * 24 + [7140] * 24 + [120445], (9.870, 12.479, 21.141))]


@pytest.fixture(scope="module")
def shape(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("shape")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run([cxx, "-O1", "-std=c++17", f"-I{CSRC}", str(d / "main.cpp"), "-o", str(d / "shape")], check=True, timeout=300)
    return lambda rows, resident: int(subprocess.run([str(d / "shape"), *map(str, [*resident, *rows])], check=True, capture_output=True).stdout)


@pytest.mark.parametrize("rows,ms", MEASURED)
def test_measured_batches(shape, rows, ms):
    t = ms[shape(rows, (7, 15, 33))]
    assert t <= 1.05 * ms[0 if len(rows) <= 7 else 1 if len(rows) <= 30 else 2]
    large = sum(n > 7 * min(rows) for n in rows)
    if 0 < large < len(rows):
        assert t <= 1.05 * min(ms)


def test_sizes_that_do_not_fit(shape):
    assert shape([2344] * 4, (0, 15, 33)) == 1 and shape([2344] * 4, (0, 0, 1)) == 2 and shape([2344], (0, 0, 0)) == -1
