"""gls_block_match_tiles: the variant that each level size met was launched
with, in a process of its own (the choice is read once)."""
import json
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]

_SCRIPT = r"""
import json
import glasscamerapublic_b200 as g
from glasscamerapublic_b200 import RawConverter, scene
c = RawConverter(0)
for w, h in ((256, 192), (336, 250)):
    wl = scene.Workload("t", w, h, levels=3, gain=1.2, read=3.0, iso=800, seed=7)
    c.demosaic(scene.make_raw(wl)[0], scene.make_params(wl), fp16=True)
print(json.dumps(g.block_match_tiles()))
c.close()
"""


@pytest.mark.parametrize("tile,code", [(None, 82), (162, 162), (44, 44), (8, 84)])
def test_every_level_size_is_listed_with_its_variant(tile, code):
    env = {k: v for k, v in os.environ.items() if k != "GLS_BM_TILE"}
    if tile:
        env["GLS_BM_TILE"] = str(tile)
    out = subprocess.run([sys.executable, "-c", _SCRIPT], cwd=ROOT, env=env, check=True, timeout=300,
                         capture_output=True, text=True).stdout
    sizes = [(256 >> l, 192 >> l) for l in range(3)] + [(336 >> l, 250 >> l) for l in range(3)]
    assert {tuple(t) for t in json.loads(out.splitlines()[-1])} == {(w, h, code) for w, h in sizes}
