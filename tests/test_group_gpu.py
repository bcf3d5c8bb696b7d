"""llava_session_group: one decoding step for several sessions with one pass over the weights.

Every member has its own prompt, position and caches; the group step must give each member what its own
llava_session steps give it.  The group runs the batched (tcgen05) products, so it is held to the same bounds as a
prompt evaluated in batches: with exact weight tiles the decode tolerance (1e-2 / 1e-3) and identical greedy tokens,
with the default fast tiles rel-L2 <= 3e-3 and the same token unless the oracle's two best logits are closer than the
logits differ.  The per-member references are the oracle's trajectories.
"""
import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

import quant_np as qn
from test_e2e_gpu import FAST_PROMPT_REL_L2, LOGIT_REL_L2, OracleSession, assert_logits_close, same_choice

pytestmark = pytest.mark.gpu

PROMPTS = [(5, 11), (9, 22), (16, 33), (3, 44), (12, 55), (7, 66), (20, 77)]       # (length, seed) per member
N_STEPS = 6


def prompt_of(n, seed):
    return [int(t) for t in np.random.default_rng(seed).integers(3, 32000, n)]


@pytest.fixture(scope="module")
def world(pkg, tmp_path_factory):
    path = str(tmp_path_factory.mktemp("group") / "tiny.bin")
    pkg.write_synthetic_model(path, "7b", n_layers=2, wtype=qn.Q4_0)
    want = []
    for n, seed in PROMPTS:
        orc = OracleSession(path)
        for t in prompt_of(n, seed):
            orc.push(t)
        logits, toks = [], []
        for _ in range(N_STEPS + 1):
            logits.append(orc.eval())
            toks.append(int(orc.argmax()))
            orc.push(toks[-1])
        orc.close()
        want.append((toks, logits))
    ctx = pkg.HostContext(path, 0)
    yield dict(ctx=ctx, want=want, vocab=32000)
    ctx.close()


def start_members(world, count):
    """Sessions that have evaluated their prompts and hold their first greedy token as the one pending token."""
    sessions = []
    for i in range(count):
        n, seed = PROMPTS[i]
        s = world["ctx"].session()
        s.set_deterministic(True)
        for t in prompt_of(n, seed):
            assert s.push_token(t)
        tok = s.predict_next_token()
        assert tok == world["want"][i][0][0]
        assert s.push_token(tok)
        sessions.append(s)
    return sessions


@pytest.mark.parametrize("count", [2, 7])
@pytest.mark.parametrize("form", ["exact", "fast"])
def test_group_steps_give_every_member_its_own_trajectory(pkg, world, form, count):
    world["ctx"].set_exact_batched_products(form == "exact")
    sessions = start_members(world, count)
    group = pkg.SessionGroup(world["ctx"], sessions)
    rel_l2 = LOGIT_REL_L2 if form == "exact" else FAST_PROMPT_REL_L2
    alive = [True] * count
    for step in range(1, N_STEPS):
        toks = group.step()
        assert toks is not None
        for i, s in enumerate(sessions):
            if not alive[i]:
                assert s.push_token(toks[i])
                continue
            want_toks, want_logits = world["want"][i]
            got = group.logits(i, world["vocab"])
            assert_logits_close(got, want_logits[step], rel_l2)
            assert same_choice(toks[i], got, want_logits[step])
            if form == "exact":
                assert toks[i] == want_toks[step]
            if toks[i] != want_toks[step]:
                alive[i] = False                  # a near-tie went the other way: this member's trajectory parts here
            assert s.push_token(toks[i])
    world["ctx"].set_exact_batched_products(False)
    # positions and token buffers are the members' own: every member evaluated prompt + N_STEPS - 1 tokens
    for i, s in enumerate(sessions):
        assert s.tokens_in_gpu() == PROMPTS[i][0] + N_STEPS - 1 and len(s.tokens()) == PROMPTS[i][0] + N_STEPS
    assert group.kernel_launches() == 1 + 2 * 9 + 2 + 1
    # a member goes on by itself from where the group left it (per-token kernels, its own recorded step)
    if form == "exact":
        s = sessions[1]
        assert s.predict_next_token() == world["want"][1][0][N_STEPS]
    group.close()
    for s in sessions:
        s.close()


def test_group_generates_on_the_device_like_step_by_step(pkg, world):
    world["ctx"].set_exact_batched_products(True)
    a = start_members(world, 3)
    ga = pkg.SessionGroup(world["ctx"], a)
    stepwise = [[] for _ in a]
    for _ in range(4):
        toks = ga.step()
        for i, s in enumerate(a):
            stepwise[i].append(toks[i])
            assert s.push_token(toks[i])
    b = start_members(world, 3)
    gb = pkg.SessionGroup(world["ctx"], b)
    assert gb.generate_greedy_on_device(4) == stepwise
    world["ctx"].set_exact_batched_products(False)
    for i, s in enumerate(b):
        assert s.tokens() == a[i].tokens() and s.tokens_in_gpu() == a[i].tokens_in_gpu()
    for g in (ga, gb):
        g.close()
    for s in a + b:
        s.close()


def test_group_refuses_what_it_cannot_do(pkg, world):
    ctx = world["ctx"]
    s = start_members(world, 2)
    with pytest.raises(RuntimeError):
        pkg.SessionGroup(ctx, s[:1])                     # one session is not a group
    with pytest.raises(RuntimeError):
        pkg.SessionGroup(ctx, [s[0], s[0]])              # the same session twice
    g = pkg.SessionGroup(ctx, s)
    assert g.step() is not None
    assert g.step() is None                              # nothing pending: the members' tokens were not pushed
    g.close()
    for x in s:
        x.close()


def test_group_members_that_sample_draw_with_their_own_sampler(pkg, world):
    """Members set to the reference's sampler (its default) get their token from the device sampler at the end of the
    group step: with the same seed a member draws the same tokens in a group as alone (exact weight tiles; the draw
    depends on the logits through the kept set and the cumulative mass, so the comparison allows a member to part from
    its lone trajectory where a probability sits within the logits' tolerance of the cut), greedy members beside them
    stay greedy, and mu moves."""
    world["ctx"].set_exact_batched_products(True)

    def members(sampled):
        out = []
        for i in range(3):
            n, seed = PROMPTS[i]
            s = world["ctx"].session()
            s.set_deterministic(i == 2 or not sampled)          # member 2 stays greedy
            s.set_seed(1000 + i)
            for t in prompt_of(n, seed):
                assert s.push_token(t)
            tok = s.predict_next_token()
            assert tok != pkg.NO_TOKEN and s.push_token(tok)
            out.append(s)
        return out

    alone = members(True)
    lone_tokens = [[s.tokens()[-1]] for s in alone]
    for _ in range(5):
        for i, s in enumerate(alone):
            tok = s.predict_next_token()
            assert s.push_token(tok)
            lone_tokens[i].append(tok)
    grouped = members(True)
    g = pkg.SessionGroup(world["ctx"], grouped)
    group_tokens = [[s.tokens()[-1]] for s in grouped]
    for _ in range(5):
        toks = g.step()
        assert toks is not None and all(t < world["vocab"] for t in toks)
        for i, s in enumerate(grouped):
            assert s.push_token(toks[i])
            group_tokens[i].append(toks[i])
    world["ctx"].set_exact_batched_products(False)
    assert g.kernel_launches() == 1 + 2 * 9 + 2 + 1 + 2                  # two sampler launches
    assert group_tokens[2] == lone_tokens[2] == world["want"][2][0][:6]   # the greedy member
    agree = [next((j for j, (a, b) in enumerate(zip(group_tokens[i], lone_tokens[i])) if a != b), 6) for i in range(2)]
    assert min(agree) >= 3 and max(agree) == 6, (group_tokens, lone_tokens)
    for i in range(2):
        assert grouped[i].mirostat_mu() != pytest.approx(10.0)           # moved from its start value (2 tau)
    g.close()
    for s in alone + grouped:
        s.close()


FAILING_LAUNCH = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stdlib.h>
/* stands in front of liblv_b200.so: refuses one graph launch, and looks whether a feed follows another one that was not waited for */
int refuse, early;
static int unread;
static void* real(const char* name) { return dlsym(dlopen(getenv("LV_REAL"), RTLD_LAZY | RTLD_NOLOAD), name); }
int lv_graph_launch(void* c, void* g) {
    if (refuse) { refuse = 0; return 1; }
    return ((int (*)(void*, void*))real("lv_graph_launch"))(c, g);
}
int lv_stream_sync(void* c, int ms) { unread = 0; return ((int (*)(void*, int))real("lv_stream_sync"))(c, ms); }
int lv_group_feed(void* c, const void* m, const void* feed, unsigned n, unsigned places) {
    early += unread;
    unread = 1;
    return ((int (*)(void*, const void*, const void*, unsigned, unsigned))real("lv_group_feed"))(c, m, feed, n, places);
}
"""
FAILING_STEP = """
import ctypes as C, os, sys
sys.path.insert(0, os.path.dirname(sys.argv[1]))
from conftest import load_pkg
pkg = load_pkg()
front = C.CDLL(os.environ["LD_PRELOAD"])
ctx = pkg.HostContext(sys.argv[2], 0)
members = []
for i in range(3):
    s = ctx.session()
    s.set_deterministic(True)
    for t in range(5 + i):
        assert s.push_token(100 * i + t)
    tok = s.predict_next_token()
    assert s.push_token(tok)
    members.append(s)
group = pkg.SessionGroup(ctx, members)
steps = []
for fail in (False, True, False):
    C.c_int.in_dll(front, "refuse").value = int(fail)
    steps.append(group.step())
    if steps[-1] is not None and len(steps) == 1:
        assert all(s.push_token(t) for s, t in zip(members, steps[-1]))
assert steps[0] is not None and steps[1] is None and steps[2] is not None
assert C.c_int.in_dll(front, "early").value == 0, "the feed was written while a launch could read it"
group.close()
"""


def test_a_step_after_a_refused_launch_waits_for_its_feed(tmp_path, pkg):
    source, front, child, path = (str(tmp_path / n) for n in ("front.c", "front.so", "child.py", "tiny.bin"))
    open(source, "w").write(FAILING_LAUNCH)
    open(child, "w").write(FAILING_STEP)
    subprocess.check_call(["gcc", "-shared", "-fPIC", "-o", front, source, "-ldl"])
    pkg.write_synthetic_model(path, "7b", n_layers=1, wtype=qn.Q4_0)
    env = dict(os.environ, LD_PRELOAD=front, LV_REAL=os.path.join(os.path.dirname(pkg.__file__), "liblv_b200.so"))
    done = subprocess.run([sys.executable, child, os.path.abspath(__file__), path], env=env, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]


@pytest.mark.parametrize("n", [1, 2, 33, 64])
def test_group_feed_sets_tokens_and_moved_positions(gpu, pkg, n):
    """lv_group_feed: tokens at their places of the members' logs, position words of moved members only."""
    cap, lib, h = 9, gpu.lib, gpu.handle
    words = gpu.upload(np.full(n * (4 + cap + 1), 7, np.uint32))                     # per member: pos[4], log[cap], a guard
    base = words.value if hasattr(words, "value") else int(words)
    members = np.zeros((n, 4), np.uint64)
    members[:, 2] = base + np.arange(n, dtype=np.uint64) * (4 * (5 + cap))
    members[:, 3] = members[:, 2] + 16
    table = gpu.upload(members)
    host = C.c_void_p()
    pkg.check(lib.lv_host_alloc(h, 12 * n, C.byref(host)))
    feed = np.ctypeslib.as_array(C.cast(host, C.POINTER(C.c_uint32)), (n, 3))
    feed[:] = [(z % cap, 100 + z, z % 3 == 0) for z in range(n)]
    pkg.check(lib.lv_group_feed(h, table, host, n, cap))
    gpu.sync()
    want = np.full((n, 5 + cap), 7, np.uint32)
    for z, (at, token, move) in enumerate(feed.tolist()):
        want[z, 4 + at] = token
        if move:
            want[z, :4] = at
    assert np.array_equal(gpu.download(words, np.uint32, want.size).reshape(want.shape), want)
    assert lib.lv_group_feed(h, table, host, 65, cap) == pkg.LV_ERR_BAD_ARGUMENTS
    pkg.check(lib.lv_host_free(h, host))
