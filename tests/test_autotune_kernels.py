"""The autotuner's cache belongs to the kernels that were measured."""
import json
import shutil

from test_autotune import _FakeBatch


def test_choices_of_other_kernels_are_not_found(tmp_path):
    from elastic_fm_vp_vs_rho_b200 import autotune
    grids = [(128, 128, 96, 10), (64, 64, 64, 10)]
    key = json.loads(autotune.batch_key(_FakeBatch(grids)))
    # entries of earlier releases: device and grids alone
    old = json.dumps({k: key[k] for k in ("device", "grids")}, sort_keys=True)
    cache = str(tmp_path / "tune.json")
    autotune.save_cache({old: {"rows": 1, "ring": 4, "ychunk": 16, "ms": 1.0}}, cache)
    assert autotune.batch_key(_FakeBatch(grids)) not in autotune.load_cache(cache)
    # a change in any of the kernels' sources or the launch rules
    for name in ("efm_stream.cu", "efm_stream.cuh", "efm_tma.cuh", "efm_internal.cuh", "efm_capi.cu"):
        csrc = tmp_path / name.replace(".", "_")
        shutil.copytree(autotune.CSRC, csrc)
        assert autotune.kernels(csrc) == key["kernels"]
        with open(csrc / name, "a") as f:
            f.write("\n")
        assert autotune.kernels(csrc) != key["kernels"]


def test_candidates_include_the_rule_and_short_chunks():
    from elastic_fm_vp_vs_rho_b200 import autotune
    chunks = {yc for _, _, yc in autotune.DEFAULT_CANDIDATES}
    assert 0 in chunks and any(0 < yc <= 5 for yc in chunks)
