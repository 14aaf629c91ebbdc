"""Plan.autotune with a cache file, on a stand-in library: no GPU.  A setting is
taken from the file only if the present kernels were timed for it."""
import json

from fame import Plan
from fame import _lib as L
from fame import plan as P


class FakeLib:
    timed = 0

    def fame_autotune(self, h, prec, nvec, chunk, tpb, us):
        self.timed += 1
        chunk._obj.value, tpb._obj.value, us._obj.value = 4, 0, 12.5
        return L.FAME_OK

    def fame_get_tune(self, h, prec, nvec, chunk, tpb, lanes):
        lanes._obj.value = -1
        return L.FAME_OK


def fake_plan():
    p = Plan.__new__(Plan)
    p.n, p.nk, p._h, p._lib = 24, 8, None, FakeLib()
    p.installed = []
    p._stream = lambda: None
    p.set_tune = lambda *a: p.installed.append(a)
    return p


def test_settings_of_older_kernels_are_timed_again(tmp_path, monkeypatch):
    path = str(tmp_path / "tune.json")
    p = fake_plan()
    first = p.autotune(cache=path)
    assert not first["cached"] and p._lib.timed == 1
    again = p.autotune(cache=path)  # the same kernels: installed
    assert again["cached"] and p._lib.timed == 1 and p.installed == [(L.FAME_C64, 8, 4, 0, -1)]
    # an entry under the key that the first kernels wrote
    (key, entry), = json.load(open(path)).items()
    old = {key.split("|kernels=")[0]: dict(entry, chunk=0, stencil_tpb=256, lanes=5)}
    json.dump(old, open(path, "w"))
    q = fake_plan()
    assert not q.autotune(cache=path)["cached"] and q._lib.timed == 1 and not q.installed
    kept = json.load(open(path))
    assert len(kept) == 2 and all(kept[k] == v for k, v in old.items())  # other entries stay
    # and one of a later generation than its own
    monkeypatch.setattr(P, "TUNED_KERNELS", P.TUNED_KERNELS + 1)
    r = fake_plan()
    assert not r.autotune(cache=path)["cached"]
