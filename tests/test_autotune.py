"""The tuner times only what it chooses between: a class that one CTA ranks has
no rulers, and what a sweep finds there is noise (128 and 96 had been kept)."""
from __future__ import annotations

import json
import re
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_classes_without_rulers_keep_their_values():
    from kascade_b200 import autotune

    src = (ROOT / "kascade_b200" / "csrc" / "ranker.cuh").read_text()
    assert autotune.ONE_CTA_MAX == int(re.search(r"ONE_CTA_MAX = (\d+);", src).group(1))
    text = (ROOT / "kascade_b200" / "csrc" / "tuned_classes.h").read_text()
    built = {k: [int(v) for v in re.findall(r"(\d+)u", re.search(rf"KS_TUNED_{k} {{(.*?)}}", text).group(1))]
             for k in ("SPACING", "SPACING_SINGLE", "BLOCK")}
    run = json.loads((ROOT / "kascade_b200" / "tuning" / "b200.json").read_text())["classes"]
    assert [autotune.uses_rulers(k) for k in range(len(run))] == [False] * 2 + [True] * 6
    for k, c in enumerate(run):
        if not autotune.uses_rulers(k):
            assert (c["spacing"], c["spacing_single"], c["block"]) == tuple(
                built[n][k] for n in ("SPACING", "SPACING_SINGLE", "BLOCK"))
