"""The rule that splits a batch's systems over the launch forms of the on-chip
solves (csrc/cg_onchip_tiers.h), compiled for the CPU and checked against what the
kernels need of it: every system's rows and shared memory fit its form, and where
the CTAs of a cluster own contiguous rows, no row gathers from a CTA that is not a
neighbour."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "cumat_b200" / "csrc"

DRIVER = r"""
#include "cg_onchip_tiers.h"
using namespace cmcg;
template <typename VT, int NF>
static int split(const OnchipBatch& b, const OnchipForm (&forms)[NF], int64_t* out) {
    const auto t = onchip_tiers<VT>(b, forms);
    for (size_t i = 0; i < t.size(); ++i) {
        const int64_t v[6] = {t[i].form.threads, t[i].form.ctas, t[i].form.per_sm, t[i].lo, t[i].hi, (int64_t)t[i].smem};
        for (int k = 0; k < 6; ++k) out[6 * i + k] = v[k];
    }
    return (int)t.size();
}
// kind 0: FP32 vectors, 1: FP64 vectors, 2: mixed
extern "C" int tiers(int kind, const int32_t* rows, const int32_t* reach, int32_t n_sys, int32_t first, int32_t ob,
                     int32_t sms, int nd, int margin, int val_bytes, int64_t* out) {
    const OnchipBatch b{rows, reach, n_sys, first, ob, sms, nd, margin, (size_t)val_bytes, kind == 2};
    return kind == 0 ? split<float>(b, kOnchip32, out) : kind == 1 ? split<double>(b, kOnchip64, out)
                                                                   : split<float>(b, kOnchipMix, out);
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("tiers")
    (d / "driver.cpp").write_text(DRIVER)
    cxx = "/usr/bin/g++" if Path("/usr/bin/g++").exists() else shutil.which("g++")
    so = d / "driver.so"
    r = subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-shared", "-fPIC", "-I", str(CSRC),
                        str(d / "driver.cpp"), "-o", str(so)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = C.CDLL(str(so))

    def f(kind, systems, nd, val_bytes, ob=1, sms=148, first=0):
        rows = np.array([s[0] for s in systems], np.int32)
        reach = np.array([s[1] for s in systems], np.int32)
        out = np.zeros(60, np.int64)
        ptr = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
        n = lib.tiers(kind, ptr(rows), ptr(reach), len(systems), first, ob, sms, nd, int(reach.max()), val_bytes, ptr(out))
        return [dict(zip(("threads", "ctas", "per_sm", "lo", "hi", "smem"), out[6 * i:6 * i + 6].tolist())) for i in range(n)]
    return f


def _check(kind, systems, nd, val_bytes, ob, first, tiers):
    """What the kernels need of a split; returns the rows that gather past a neighbour."""
    if not tiers:
        return
    vec = 8 if kind == 1 else 4
    slots = 8 if kind == 1 else 16
    margin = (max(s[1] for s in systems) + 3) // 4 * 4
    assert tiers[0]["lo"] == first * ob and tiers[-1]["hi"] == len(systems) * ob
    assert all(a["hi"] == b["lo"] for a, b in zip(tiers, tiers[1:]))
    for t in tiers:
        # 227 KB of a CTA and 228 KB of an SM hold the dynamic and the static arrays
        # and 1 KB per CTA for the system
        if kind == 1 or (kind == 2 and t["threads"] == 256):
            static = 2 * 128 * 8 + 16 if kind == 1 else 1040
            assert t["smem"] + static <= 227 * 1024 and t["per_sm"] * (t["smem"] + static + 1024) <= 228 * 1024, t
        else:   # groups share one CTA's memory, each with its scratch before its part
            scratch, static = (544, 528) if kind == 0 else (1056, 1040)
            part = -(-t["smem"] // 16) * 16 + (scratch if t["per_sm"] > 1 else 0)
            assert -(-part * t["per_sm"] // 64) * 64 + static <= 227 * 1024, t
    for t in tiers:
        per = t["threads"] * t["ctas"]
        for n, reach in systems[t["lo"] // ob:t["hi"] // ob]:
            nk = (-(-n // per) + 1) // 2 * 2
            assert nk <= slots
            own = nk * t["threads"]
            pair = kind == 0 and t["ctas"] == 2
            assert ((2 * own if pair else own) + 2 * margin) * vec + own * nd * val_bytes <= t["smem"]
            if t["ctas"] > 1 and not pair:
                # contiguous rows: CTA r // own owns row r
                r = np.arange(n)
                for o in (reach, -reach):
                    ok = (r + o >= 0) & (r + o < n)
                    assert np.all(np.abs((r[ok] + o) // own - r[ok] // own) <= 1), (n, reach, t)


# the batches with a long grid or a band among squares; (rows, largest offset) by size
LONG = [(1, [(10000, 100)] * 10 + [(4400, 2200)] + [(3600, 60)] * 2, 5, 8),
        (1, [(13000, 1300), (10500, 3500), (9000, 900)], 7, 4), (1, [(13000, 1300), (10500, 3500), (9000, 900)], 7, 2),
        (1, [(16384, 128)] * 10 + [(5000, 3500)], 5, 4), (1, [(14770, 2110)] * 200, 5, 8)]


@pytest.mark.parametrize("case", range(len(LONG)))
def test_halo_of_every_system(rule, case):
    kind, systems, nd, vb = LONG[case]
    for sms in (1, 148):
        _check(kind, systems, nd, vb, 1, 0, rule(kind, systems, nd, vb, sms=sms))


@pytest.mark.parametrize("kind", [0, 1, 2])
def test_random_batches(rule, kind):
    rng = np.random.RandomState(kind)
    found = 0
    for trial in range(4000):
        nd = int(rng.choice([5, 7]))
        top = 8192 if kind == 2 else 16384
        systems = []
        for _ in range(rng.randint(1, 7)):
            n = int(np.exp(rng.uniform(0, np.log(top))))
            reach = int(rng.choice([min(n - 1, int(n ** 0.5)), rng.randint(0, n), min(n - 1, rng.randint(1, 40))]))
            systems += [(n, reach)] * int(rng.choice([1, 1, 2, 60]))
        systems.sort(key=lambda s: -s[0])
        # (the order goes by entries, so a band with fewer diagonals may stand behind smaller systems)
        if rng.rand() < 0.3:
            i = rng.randint(len(systems))
            systems.insert(rng.randint(len(systems)), systems.pop(i))
        ob, vb = int(rng.choice([1, 3])), int(rng.choice([2, 4, 8]))
        tiers = rule(kind, systems, nd, vb, ob=ob)
        found += bool(tiers)
        _check(kind, systems, nd, vb, ob, 0, tiers)
    assert found > 400   # (the rule does give forms)
