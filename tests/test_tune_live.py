"""The tuner times only knobs that change a launch: without one it makes no
medium and no run, stores an empty setting and still reads and applies
settings saved before."""

from pmmoto_gb300 import tune


def test_nothing_is_timed_without_a_live_knob(tmp_path, monkeypatch):
    from pmmoto_gb300.domain_generation import grf

    def no_medium(*a, **k):
        raise AssertionError("a medium was generated")

    monkeypatch.setenv("PMG_TUNE_CACHE", str(tmp_path / "c.json"))
    monkeypatch.delenv("PMG_TUNE", raising=False)
    monkeypatch.setattr(tune, "gpu_name", lambda: "cpu")
    monkeypatch.setattr(grf, "gen_grf_medium", no_medium)
    monkeypatch.setattr(tune, "_time", no_medium)
    try:
        for fn, kernel in ((tune.tune_edt, "edt"), (tune.tune_cc, "cc")):
            assert set(tune.KNOBS[kernel]) <= tune.INERT
            for force in (False, True):
                assert fn((64, 64, 64), force=force) == {}
            assert tune.load_cache()[tune.key(kernel, (64, 64, 64))] == {"settings": {}, "ms": {}}
    finally:
        tune._applied.clear()


def test_saved_settings_of_former_knobs_still_load(tmp_path, monkeypatch):
    monkeypatch.setenv("PMG_TUNE_CACHE", str(tmp_path / "c.json"))
    monkeypatch.delenv("PMG_TUNE", raising=False)
    monkeypatch.setattr(tune, "gpu_name", lambda: "cpu")
    tune.save_entry(tune.key("edt", (64, 64, 64)), {"edt.pair_seg": 512}, {"edt.pair_seg": {"512": 1.0}})
    try:
        assert tune.tune_edt((64, 64, 64)) == {"edt.pair_seg": 512}
        assert tune.get_lib("edt.pair_seg") == 512
    finally:
        tune._applied.clear()
        tune.reset_lib("edt")


def test_live_knobs_are_timed(monkeypatch):
    seen = []
    monkeypatch.setattr(tune, "_time", lambda run, steps: float(seen[-1][1]))
    best, ms = tune._descend("batch", lambda: None, 1, lambda n, v: seen.append((n, v)))
    assert best == {"batch.workers": 2} and set(ms["batch.workers"]) == {"2", "4", "8", "16"}
