"""The device's pair sort through the program that writes pairs in row order:
counts around a tile of 2,048 pairs, keys of few bits (two passes at the
least) and of many, and tables of one row; every pair of the tables is one."""
import numpy as np
import pytest

import hyperblocker_gb300 as hb
from hyperblocker_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_l,n_r", [(1, 1), (1, 2), (2, 1), (1, 300), (23, 89), (2, 1024), (3, 683),
                                     (129, 257), (4099, 5), (2, 70001), (1500, 2100)])
def test_every_pair_in_row_order(built, tmp_path, n_l, n_r):
    def write(path, n):
        path.write_text("".join(f"{i},a,a,k\n" for i in range(n)))
        return str(path)

    rules = tmp_path / "rules"
    rules.mkdir()
    (rules / "0.yaml").write_text(synth.rule_yaml([3], [(1, 0.0)]))
    out = tmp_path / "pairs.csv"
    assert hb.run_cli(["run_hyperblocker_exec", "-data_l", write(tmp_path / "l.csv", n_l), "-data_r",
                       write(tmp_path / "r.csv", n_r), "-rule_dir", str(rules), "-n_partitions", "1",
                       "-o", str(out)]) == 0
    got = np.fromstring(out.read_text().replace("\n", ","), dtype=np.int64, sep=",").reshape(-1, 2)
    want = np.stack((np.repeat(np.arange(n_l), n_r), np.tile(np.arange(n_r), n_l)), 1)
    assert np.array_equal(got, want)
