"""The device-resident searcher's per-seed stages (coverage walk, evaluations, rows) where their chunks end: sites in
groups of 32, components in blocks of 256 per seed.  Every evaluation becomes a row (csv_min=0), and the files are those
of the per-stage path, whose loops run on the host."""
import collections
import json
import os

import numpy as np
import pytest

from test_search_gpu import G, same_outputs

pytestmark = pytest.mark.gpu


def finds(n):
    return [f["seed"] for f in json.load(open(os.path.join(G, "finds.json")))[:n]]


# (sites per seed, fewest evaluations that one seed must have)
@pytest.mark.parametrize("sites,most", [(300, 257), (1, 1), (32, 33), (33, 33)])
def test_every_evaluation_equals_the_per_stage_path(dsg, tmp_path, sites, most):
    seeds = finds(24)
    rows, _ = same_outputs(tmp_path, ["0", "0", "8", "stdin=1", "gpu=1", "gscan=1", "csv_min=0", f"sites={sites}"],
                           stdin="".join(f"{s}\n" for s in seeds))
    per = collections.Counter(r.split(",")[0] for r in rows)
    assert max(per.values()) >= most, max(per.values())
    dsg.scan_init_default()                              # the device path itself finished every seed: none handed back
    dsg.search_open(seeds_cap=64, csv_min=0, max_sites=sites)
    try:
        recs, drows, unf, _, _ = dsg.search_seeds(np.array([s & ((1 << 64) - 1) for s in seeds], dtype=np.uint64))
    finally:
        dsg.search_close()
    assert len(recs) == len(seeds) and len(unf) == 0
    assert len(drows) == sum(int(r["nrows"]) for r in recs)
