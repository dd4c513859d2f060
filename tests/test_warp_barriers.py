"""The barriers of the lane form's kernels, run on the host: the generated
module's own propagation and reverse-sweep kernels, compiled as C++ with one
host thread per GPU thread, a warp barrier that waits for the warp's threads
that have not returned and a CTA barrier that waits for the CTA's.  A launch in
which every thread that is left waits is a deadlock.  Lanes that stop before
the recurrences of an iteration (a stop word of their batch, a full record or
tape) and take the next lane from the queue must not part a warp."""

import ctypes
import re
import subprocess

import numpy as np
import pytest

from cuda_host import INTRINSICS
from hyk import _lib
from hyk import workloads as W
from hyk.decompose import taylor_decompose

ORDER, TPB, NE = 4, 64, 6

SHIM = r"""
#include <condition_variable>
#include <mutex>
#include <thread>
#include <vector>
struct Dim { unsigned x; };
static thread_local Dim threadIdx, blockIdx;
static const Dim blockDim = {TPB}, gridDim = {1};
static inline unsigned __ballot_sync(unsigned, bool) { return 0; }  // (kernels that are not run here)
static inline unsigned __activemask() { return 1; }
template <class T> static inline T __shfl_sync(unsigned, T v, int) { return v; }
template <class T> static inline T __ldcg(const T *p) { return *p; }
static inline void __nanosleep(unsigned) {}
static inline void __threadfence_system() {}

struct Deadlock {};
enum { RUN, WARP, CTA, GONE };
static std::mutex mx;
static std::condition_variable cv;
static int where[TPB];
static unsigned long long pass[TPB];
static bool dead;
// Releases the barriers that are complete; a deadlock when nobody runs.
static void settle() {
    bool any = false, run = false, cta = true;
    for (int w = 0; w < TPB; w += 32) {
        bool all = true, some = false;
        for (int i = w; i < w + 32; ++i) {
            some = some || where[i] == WARP;
            all = all && (where[i] == WARP || where[i] == GONE);
        }
        for (int i = w; all && some && i < w + 32; ++i)
            if (where[i] == WARP) { where[i] = RUN; ++pass[i]; any = true; }
    }
    bool some = false, left = false;
    for (int i = 0; i < TPB; ++i) {
        some = some || where[i] == CTA;
        cta = cta && (where[i] == CTA || where[i] == GONE);
    }
    for (int i = 0; cta && some && i < TPB; ++i)
        if (where[i] == CTA) { where[i] = RUN; ++pass[i]; any = true; }
    for (int i = 0; i < TPB; ++i) { run = run || where[i] == RUN; left = left || where[i] != GONE; }
    if (left && !run) { dead = true; any = true; }
    if (any) cv.notify_all();
}
static void wait_at(int kind) {
    std::unique_lock<std::mutex> lk(mx);
    const int t = (int)threadIdx.x;
    if (dead) throw Deadlock();
    where[t] = kind;
    const unsigned long long at = pass[t];
    settle();
    cv.wait(lk, [&] { return dead || pass[t] != at; });
    if (dead) throw Deadlock();
}
static inline void __syncwarp(unsigned = 0xffffffffu) { wait_at(WARP); }
static inline void __syncthreads() { wait_at(CTA); }
template <class T, class S> static inline T atomicAdd(T *p, S v) {
    std::lock_guard<std::mutex> lk(mx);
    const T o = *p;
    *p = (T)(o + (T)v);
    return o;
}
template <class T> static inline T atomicMin(T *p, T v) {
    std::lock_guard<std::mutex> lk(mx);
    const T o = *p;
    if (v < o) *p = v;
    return o;
}
template <class T, class S> static inline T atomicOr(T *p, S v) {
    std::lock_guard<std::mutex> lk(mx);
    const T o = *p;
    *p |= (T)v;
    return o;
}
template <class T> static inline T atomicCAS(T *p, T, T) { return *p; }
"""

DRIVER = r"""
// One CTA over n lanes; returns 1 when it deadlocked.
extern "C" int run(int adjoint, hyk_kparams *P) {
    std::vector<double> jets((size_t)HYK_NSLOT * HYK_STRIDE, 0.0);
    P->jets = jets.data();
    P->slot_sms = 1;
    P->slot_units = 32;
    P->slot_layers = TPB / 32;
    P->n_slots = TPB;
    dead = false;
    for (int i = 0; i < TPB; ++i) { where[i] = RUN; pass[i] = 0; }
    std::vector<std::thread> ts;
    for (unsigned t = 0; t < TPB; ++t)
        ts.emplace_back([=] {
            threadIdx.x = t;
            blockIdx.x = 0;
            try {
#ifdef HYK_ADJOINT
                if (adjoint) hyk_adjoint_kernel(*P);
                else
#endif
                    hyk_prop_kernel(*P);
            } catch (const Deadlock &) {}
            std::lock_guard<std::mutex> lk(mx);
            where[t] = GONE;
            if (!dead) settle();
        });
    for (auto &t : ts) t.join();
    return dead ? 1 : 0;
}
extern "C" void init(hyk_kparams *P) {
    for (unsigned long long l = 0; l < P->n_lanes; ++l) {
        blockIdx.x = (unsigned)(l / TPB);
        threadIdx.x = (unsigned)(l % TPB);
        hyk_prop_init_kernel(*P);
    }
}
#define FIELD(f) if (!std::strcmp(name, #f)) { std::memcpy(&P->f, &v, sizeof P->f); return 0; }
extern "C" int set(hyk_kparams *P, const char *name, unsigned long long v) {
    FIELD(n_lanes) FIELD(ld) FIELD(state) FIELD(t_hi) FIELD(t_lo) FIELD(tf_hi) FIELD(max_steps) FIELD(tc_out)
    FIELD(tc_thi) FIELD(tc_tlo) FIELD(tc_cap) FIELD(rem_hi) FIELD(rem_lo) FIELD(outcome) FIELD(min_h) FIELD(max_h)
    FIELD(n_steps) FIELD(n_iter) FIELD(last_h) FIELD(status) FIELD(iters_per_launch) FIELD(queue) FIELD(finished)
    FIELD(n_order) FIELD(ck_x) FIELD(ck_t) FIELD(ck_h) FIELD(ck_cap) FIELD(adj_steps) FIELD(adj_lambda)
    FIELD(adj_pbar) FIELD(stop_iter) FIELD(stop_group) FIELD(persistent)
    return 1;
}
extern "C" int size(void) { return (int)sizeof(hyk_kparams); }
"""


@pytest.fixture(scope="module")
def kernels(libhyk, tmp_path_factory):
    d, keep = taylor_decompose(W.kepler_sys()).as_c()
    cfg = _lib.hyk_config_t(TPB, 0, _lib.HYK_CFG_ADJOINT | _lib.HYK_CFG_GLOBAL_JETS, 0)
    buf = ctypes.create_string_buffer(1 << 24)
    assert libhyk.hyk_codegen_check(ctypes.byref(d), ORDER, ctypes.byref(cfg), 2, buf, len(buf), None, None) == 0
    src = buf.value.decode()
    assert "#define HYK_PHASE 1" in src
    src = re.sub(r"asm volatile\(.*?\);", ";", src, flags=re.S)
    tmp = tmp_path_factory.mktemp("barriers")
    f, so = str(tmp / "k.cpp"), str(tmp / "k.so")
    with open(f, "w") as fh:
        fh.write("#define TPB {}\n".format(TPB) + INTRINSICS + SHIM + src + DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-ffp-contract=off", "-shared", "-fPIC", "-pthread", f, "-o", so],
                   check=True)
    return ctypes.CDLL(so)


class _Launch:
    """A propagation's arrays and the parameter block that points to them."""

    def __init__(self, lib, state, tf, **extra):
        self.lib, n = lib, state.shape[1]
        f, i = np.float64, np.int64
        self.a = {"state": state, "tf_hi": tf, "t_hi": np.zeros(n), "t_lo": np.zeros(n), "queue": np.zeros(4, i),
                  "finished": np.zeros(4, i)}
        for k, ty in (("rem_hi", f), ("rem_lo", f), ("outcome", i), ("min_h", f), ("max_h", f), ("n_steps", i),
                      ("n_iter", i), ("last_h", f), ("status", np.uint32)):
            self.a[k] = np.zeros(n, ty)
        self.p = ctypes.create_string_buffer(lib.size())
        for k, v in {**self.a, "n_lanes": n, "ld": n, "n_order": n, "iters_per_launch": (1 << 64) - 1, "persistent": 1,
                     **extra}.items():
            self.set(k, v)
        lib.init(self.p)

    def set(self, name, v):
        if isinstance(v, np.ndarray):
            self.a[name] = v
            v = v.ctypes.data
        assert self.lib.set(self.p, name.encode(), ctypes.c_ulonglong(v)) == 0

    def run(self, adjoint=0):
        self.a["queue"][:] = 0
        return self.lib.run(adjoint, self.p)


N = 151
DONE, STOPPED, CAPACITY = 1, 2, 4


def _ics(seed=3):
    rng = np.random.default_rng(seed)
    return np.ascontiguousarray(W.kepler_ics(N, seed=seed)), rng.uniform(0.05, 2.0, N)


@pytest.mark.parametrize("persistent", [1, 0])
def test_finite_lanes(kernels, persistent):
    st, tf = _ics()
    ref = st.copy()
    L = _Launch(kernels, st, tf, persistent=persistent, iters_per_launch=(1 << 64) - 1 if persistent else 1)
    for _ in range(1 if persistent else 200):
        assert L.run() == 0
        if not persistent and (L.a["status"] & DONE).all():
            break
    assert (L.a["status"] == DONE).all() and np.array_equal(L.a["t_hi"], tf)
    assert len(np.unique(L.a["n_iter"])) > 3 and not np.array_equal(st, ref)


@pytest.mark.parametrize("bad", [[0], [40], [150], [7, 63, 100]])
@pytest.mark.parametrize("group", [0, 4, 32])
def test_lanes_that_stop_with_their_batch(kernels, group, bad):
    """A state that becomes non-finite lowers its group's stop word while the
    group's other lanes are at other iterations."""
    st, tf = _ics()
    st[0, bad] = np.nan
    stop = np.full(1 if group == 0 else (N + group - 1) // group, (1 << 64) - 1, np.uint64)
    L = _Launch(kernels, st, tf, stop_iter=stop, stop_group=group)
    assert L.run() == 0
    assert (L.a["status"] & (DONE | STOPPED) != 0).all()
    g = np.arange(N) // (group or N)
    assert (stop[np.unique(g[bad])] == 1).all()


@pytest.mark.parametrize("cap", [1, 2, 3, 5])
@pytest.mark.parametrize("kind", ["tape", "record"])
def test_lanes_that_fill_their_store(kernels, kind, cap):
    st, tf = _ics()
    if kind == "tape":
        extra = dict(ck_x=np.zeros((cap, NE, N)), ck_t=np.zeros((cap, N)), ck_h=np.zeros((cap, N)), ck_cap=cap)
    else:
        extra = dict(tc_out=np.zeros((cap, NE, ORDER + 1, N)), tc_thi=np.zeros((cap, N)), tc_tlo=np.zeros((cap, N)),
                     tc_cap=cap)
    L = _Launch(kernels, st, tf, **extra)
    assert L.run() == 0
    full = (L.a["status"] & CAPACITY) != 0
    assert full.any() and (L.a["n_iter"][full] == cap).all() and ((L.a["status"] & DONE != 0) | full).all()


def test_reverse_sweep_of_uneven_tapes(kernels):
    st, tf = _ics()
    x0 = st.copy()
    cap = 64
    ck = dict(ck_x=np.zeros((cap, NE, N)), ck_t=np.zeros((cap, N)), ck_h=np.zeros((cap, N)), ck_cap=cap)
    L = _Launch(kernels, st, tf, **ck)
    assert L.run() == 0 and (L.a["status"] == DONE).all()
    lam, pb = np.random.default_rng(1).normal(size=(NE, N)), np.zeros((1, N))
    l0 = lam.copy()
    L.set("adj_steps", L.a["n_iter"])
    L.set("adj_lambda", lam)
    L.set("adj_pbar", pb)
    assert L.run(adjoint=1) == 0
    # each lane alone in its launch: the same bits
    for b in range(0, N, 10):
        one = dict((k, np.ascontiguousarray(ck[k][..., b:b + 1])) for k in ("ck_x", "ck_t", "ck_h"))
        D = _Launch(kernels, np.ascontiguousarray(x0[:, b:b + 1]), tf[b:b + 1].copy(), ck_cap=cap, **one)
        lb = np.ascontiguousarray(l0[:, b:b + 1])
        D.set("adj_steps", L.a["n_iter"][b:b + 1].copy())
        D.set("adj_lambda", lb)
        D.set("adj_pbar", np.zeros((1, 1)))
        assert D.run(adjoint=1) == 0 and np.array_equal(lb[:, 0], lam[:, b])
