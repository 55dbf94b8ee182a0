"""A tile choice is read back only by the kernels it was measured with: a cache file written before the bucketing
changed (keys without a kernel number, or with an older one) is measured again, and its entries stay in the file."""
import json

import pytest

from gbpowspec import tune


@pytest.mark.parametrize("suffix", ["", f"|k{tune.KERNELS - 1}"])
def test_choices_of_other_kernels_are_measured_again(tmp_path, suffix):
    path = tmp_path / "tiles.json"
    old = "GB300|N512|tsc|G2|n2^22" + suffix
    path.write_text(json.dumps({old: {"tiles": [8, 4], "ms": {"8x4": 1.0, "4x4": 2.0}}}))
    calls = []

    def timer(N, mas, interlace, n, tiles, device):
        calls.append(tiles)
        return {(8, 4): 1.9e-3, (4, 4): 1.6e-3}[tiles]
    t = tune.Tuner(path=str(path), timer=timer, variants=lambda N: [(8, 4), (4, 4)], device_name=lambda d: "GB300")
    assert t.best(512, "tsc", True, n=4 << 20) == (4, 4)
    assert len(calls) == 2
    assert json.loads(path.read_text())[old]["tiles"] == [8, 4]
    assert t.best(512, "tsc", True, n=4 << 20) == (4, 4) and len(calls) == 2
