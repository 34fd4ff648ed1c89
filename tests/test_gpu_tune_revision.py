"""The tuning cache: entries measured on other kernels (a file of another revision) are timed again."""
import json

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("revision", ["1", "3", "\"x\""])
def test_entries_of_another_revision_are_timed_again(tmp_path, revision):
    from mcstar_b200 import tune
    shape = (24, 20, 1)
    cache = tmp_path / "tune.json"
    opts, ms = tune(shape, np.float32, str(cache))
    text = cache.read_text()
    head, rest = text.split("\n", 1)
    current = json.loads(text)["pfc_tune"]
    (key, entry), = json.loads(text)["entries"].items()
    entry = dict(entry, radix_order=1, ms_per_step=123.5)
    cache.write_text(head.replace(str(current), revision) + "\n  \"%s\": %s\n}}\n" % (key, json.dumps(entry)))
    again, ms2 = tune(shape, np.float32, str(cache))
    assert ms2 < 10.0 * ms  # not the entry's 123.5 ms
    data = json.loads(cache.read_text())
    assert data["pfc_tune"] == current
    assert data["entries"][key]["ms_per_step"] == pytest.approx(ms2, rel=1e-4)
    # the same entry under the current revision is taken as it stands
    cache.write_text(head + "\n  \"%s\": %s\n}}\n" % (key, json.dumps(entry)))
    kept, ms3 = tune(shape, np.float32, str(cache))
    assert ms3 == pytest.approx(123.5) and kept["radix_order"] == 1
