"""Calls at the edges of what the engine and its operators take: sizes at which a product's form changes or its shared memory fills,
routings that cover a part of the experts, non-finite inputs, memory that runs out."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _cfg(F, **over):
    d = dict(n_layer=2, hidden=1024, n_expert=16, top_k=4, ffn=256, n_q_head=8, n_kv_head=1, gdn_k_head=2, gdn_v_head=4, vocab=2048, max_ctx=256, max_rows=32, attn_every=2, n_seq=1)
    d.update(over)
    return F.flash_next_config(**d)


def _engine(F, **over):
    cfg = _cfg(F, **over)
    e = F.Engine(cfg)
    e.init_synthetic(seed=3, sigma=0.02)
    return cfg, e


def _logits(e, cfg, T):
    return e.tensor("buf.logits", torch.float32, (cfg.max_rows, cfg.vocab))[:T].clone()


def test_a_window_is_complete_when_its_commit_returns(F):
    """prompt, and windows whose results are not taken: the logits are those of the last window as soon as the commit is back, read on a
    stream that knows nothing of the engine's."""
    cfg, e = _engine(F, vocab=65536, n_seq=2, max_ctx=512)
    try:
        rng = np.random.default_rng(7)
        draw = lambda n: rng.integers(0, cfg.vocab, size=n).tolist()

        def lanes():
            e.verify_lanes([0, 1], [draw(5), draw(5)], want_result=False)
            e.commit_lanes([0, 1], [5, 5])
        for warm in range(3):                        # (a window's first run is waited for: it is captured then)
            for what in (lambda: e.prompt(draw(40)), lambda: e.prefill(draw(32)), lanes):
                e.reset(0)
                e.reset(1)
                what()
                at_once = _logits(e, cfg, 1)
                torch.cuda.synchronize()
                assert torch.equal(at_once, _logits(e, cfg, 1))
    finally:
        e.close()


def test_experts_of_a_routing_that_covers_a_part(F):
    """A routing over half of the experts, or without the shared one, and moe_experts over all of them: the rows of experts that the job
    list leaves out count as zero, whatever the memory held before."""
    from test_gpu_ops import _moe_fixture
    E, H, Fn, K, T = 16, 512, 256, 4, 5
    fx = _moe_fixture(F, E, H, Fn, seed=31)
    x = torch.randn((T, H), device="cuda", generator=torch.Generator(device="cuda").manual_seed(9))
    w = (fx["gu_t"], fx["dn_t"], fx["sh_gu_t"], fx["sh_dn_t"])
    P = T * K + T
    for rng, shared in (((0, E // 2), True), ((0, E), False), ((0, 0), True)):
        route = F.router_route(fx["wr"], x, K, e_lo=rng[0], e_hi=rng[1], add_shared=shared)
        want, hw, pw = F.moe_experts(*w, route, x, Fn, K, e_lo=rng[0], e_hi=rng[1], add_shared=shared)
        dirt = [torch.full((P, n), float("nan"), device="cuda") for n in (Fn, H, Fn, H)]
        del dirt                                     # (the caching allocator hands this memory out again)
        got, h, part = F.moe_experts(*w, route, x, Fn, K)
        assert torch.equal(got, want) and torch.equal(h, hw) and torch.equal(part, pw), (rng, shared)


ASKED = {"gate|up": ["l0.experts_gu", "l1.experts_gu"], "down": ["l0.experts_dn", "l1.experts_dn"], "projections": ["l0.w_in", "l1.w_out", "mtp.fc_hid"],
         "heads and one layer": ["head", "l1.w_in", "l1.experts_gu", "l1.experts_dn", "l1.shared_dn"]}


@pytest.mark.parametrize("asked", sorted(ASKED))
def test_engines_with_some_matrices_in_the_interchange_layout(F, asked):
    """Matrices that were asked for by name among others that were not: windows, drafts and prompts take each from where it is, in one chain of
    kernels that overlap.  The two layouts part by the order of f32 sums and by rows whose codes move one step (1 / 65,024 of a block's
    largest value); a prompt's rows are rounded to f16 three times a layer (2^-11 each).  With routers of zeros no near tie parts them."""
    toks = np.random.default_rng(8).integers(0, 2048, size=400).tolist()
    got = []
    for names in ([], ASKED[asked]):
        cfg, e = _engine(F, max_ctx=512)
        try:
            for n in names:
                e.tensor(n, torch.uint8)
            for l in ("l0.", "l1.", "mtp."):
                e.tensor(l + "router", torch.float32)[:cfg.n_expert * cfg.hidden] = 0.0
            torch.cuda.synchronize()
            r = []
            for T in (1, 5, 20):
                for _ in range(3):                   # (the first run, the captured one, and that again)
                    e.verify(toks[:T])
                    r.append(_logits(e, cfg, T))
            assert torch.equal(r[-1], r[-2])
            e.commit([0])
            r.append(torch.tensor(e.draft(3), device="cuda"))
            for n in (12, 30, 380):
                e.reset()
                e.prompt(toks[:n])
                r.append(_logits(e, cfg, 1))
            got.append(r)
            assert e.error_bits() == 0
        finally:
            e.close()
    for i, (a, b) in enumerate(zip(*got)):
        tol = 3e-4 if i < 9 else 3 * 2.0 ** -11
        assert torch.equal(a, b) if i == 9 else float((a - b).norm() / b.norm()) < tol, i


@pytest.mark.parametrize("name", ["l0.shared_gu", "l0.shared_dn"])
def test_a_matrix_asked_for_when_its_partner_finds_no_memory(F, name):
    """The shared expert's matrix moves to the interchange layout together with the stack of routed ones.  Where that finds no room the
    call fails and nothing has moved: the same window and prompt give the same bits."""
    cfg, e = _engine(F, n_layer=1, hidden=2048, ffn=512, n_expert=512)
    try:
        toks = np.random.default_rng(9).integers(0, cfg.vocab, size=40).tolist()

        def passes():
            e.reset()
            e.verify(toks[:5])
            w = _logits(e, cfg, 5)
            e.commit([0])
            e.draft(2)
            e.reset()
            e.prompt(toks)
            return w, _logits(e, cfg, 1)
        want, held = passes(), e.device_bytes()
        torch.cuda.empty_cache()
        room = 64 << 20                              # the shared matrices take 1 MB, the stacks 231 and 461
        fill = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda")
        with pytest.raises(KeyError):
            e.tensor(name, torch.uint8)
        del fill
        torch.cuda.empty_cache()
        assert e.device_bytes() == held
        assert all(torch.equal(a, b) for a, b in zip(passes(), want))
        size = e.tensor(name, torch.uint8).numel()   # with the memory back it is handed out
        assert size == (F.iq3s_bytes(1024, 2048) if name.endswith("gu") else F.iq3s_bytes(2048, 512))
    finally:
        e.close()


@pytest.mark.parametrize("hidden,vocab", [(1024, 131072), (2048, 151936)])
def test_a_row_of_a_large_head_gives_the_same_bits_in_any_window(F, hidden, vocab):
    """A head of more than 64 MB (1,024 columns: 27 or 28 units a block; 2,048: 32 or 33): a row's logits are the same bits alone, among
    eight rows, nine, twenty and thirty-two, whatever form of the product those take."""
    cfg, e = _engine(F, hidden=hidden, vocab=vocab)
    try:
        toks = np.random.default_rng(2).integers(0, cfg.vocab, size=32).tolist()
        e.verify(toks)
        every = _logits(e, cfg, 32)
        for T in (1, 4, 8, 9, 12, 16, 20, 24):
            e.verify(toks[:T])
            assert torch.equal(_logits(e, cfg, T), every[:T]), T
    finally:
        e.close()


@pytest.mark.parametrize("hidden", [3072, 3584, 4096])
def test_a_large_head_over_wide_rows(F, hidden):
    """A vocabulary head of more than 64 MB over rows of up to 4,096 columns, at every number of row groups: the rows' images and the tiles
    in flight share a block's memory.  A row's logits are the same bits in all of them."""
    cfg, e = _engine(F, hidden=hidden, vocab=40960, n_expert=4, top_k=2)
    try:
        toks = np.random.default_rng(1).integers(0, cfg.vocab, size=32).tolist()
        e.verify(toks)
        every = _logits(e, cfg, 32)
        assert bool(torch.isfinite(every).all())
        for T in (1, 5, 8, 13, 17, 20):
            e.verify(toks[:T])
            assert torch.equal(_logits(e, cfg, T), every[:T]), T
    finally:
        e.close()


@pytest.mark.parametrize("top_k,T", [(15, 32), (16, 29), (16, 32), (32, 15), (32, 32)])
def test_wide_windows_of_many_picks(F, top_k, T):
    """Up to 32 picks for each of 32 rows: the job list (40 bytes a job) shares a block's memory with the tiles in flight.  Against the
    same rows one at a time: bit for bit."""
    cfg, e = _engine(F, hidden=2048, n_expert=64, top_k=top_k)
    try:
        toks = np.random.default_rng(3).integers(0, cfg.vocab, size=T).tolist()
        e.verify(toks)
        every = _logits(e, cfg, T)
        for t in range(3):
            e.verify([toks[t]])
            assert torch.equal(_logits(e, cfg, 1)[0], every[t]), t
            e.commit([0])
    finally:
        e.close()


def test_a_tree_commit_without_attention_layers(F):
    """Every layer a DeltaNet (attn_every above the layer count): a path that is no prefix moves the device's position on by its rows, once."""
    cfg, e = _engine(F, attn_every=5)
    try:
        pos = lambda: int(e.tensor("seq.pos", torch.int32)[0].item())
        e.verify([5, 6, 7, 8], [-1, 0, 0, 2])
        e.commit([0, 2, 3])
        torch.cuda.synchronize()
        d = e.draft(2)                               # (waits for the commit)
        assert e.pos() == 3 and pos() == 3
        e.verify([9, 10])
        e.commit([0, 1])
        e.draft(1)
        assert e.pos() == 5 and pos() == 5 and len(d) == 2
    finally:
        e.close()


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("row", [5, 8, 15, 17])
def test_a_prompts_rows_before_a_non_finite_one(F, bad, row):
    """DeltaNet over a prompt, one value of row `row` not finite: the rows before it, of its own group of eight too, keep their bits."""
    nk, nv, hs, NS, T = 2, 4, 128, 4, 21
    g = torch.Generator(device="cuda").manual_seed(4)
    rnd = lambda *s: torch.randn(s, device="cuda", generator=g)
    ch = (2 * nk + nv) * hs
    x, ab, hist, S = rnd(T, ch + nv * hs), rnd(T, 2 * nv), rnd(NS, 3, ch), 0.1 * rnd(NS, nv, hs, hs)
    convw, dt, a, nw = rnd(ch, 4), rnd(nv), -rnd(nv).abs(), rnd(hs)
    run = lambda x, ab: F.gdn_prompt(x, ab, hist.clone(), convw, dt, a, nw, S.clone(), 1, nk, nv)
    clean = run(x, ab)
    for what in ("q", "k", "v", "gate"):
        y, b = x.clone(), ab.clone()
        if what == "gate":
            b[row, 0] = bad
        else:
            y[row, {"q": 0, "k": nk * hs, "v": 2 * nk * hs}[what]] = bad
        got = run(y, b)
        assert torch.equal(got[:row], clean[:row]), what


@pytest.mark.parametrize("nq,nkv", [(16, 2), (64, 8)])
def test_many_rows_merge_to_the_bits_of_a_few(F, nq, nkv):
    """The merge of the splits in small blocks (many rows and heads) and in large ones (few)."""
    T, ctx = 32, 3000
    g = torch.Generator(device="cuda").manual_seed(10)
    qg = torch.randn((T, nq, 512), device="cuda", generator=g)
    kc, vc = (torch.randn((ctx + T, nkv, 256), device="cuda", generator=g).half() for _ in range(2))
    pos = torch.arange(ctx, ctx + T, dtype=torch.int32, device="cuda")
    every = F.attn(qg, kc, vc, pos[:1])
    for a in range(0, T, 4):
        assert torch.equal(F.attn(qg[a:a + 4].contiguous(), kc, vc, pos[a:a + 1]), every[a:a + 4]), a


@pytest.mark.parametrize("E,H,T", [(31, 2304, 33), (16, 3072, 64), (512, 4096, 49)])
@pytest.mark.parametrize("normed", [False, True])
def test_router_over_rows_of_more_than_2048_columns(F, E, H, T, normed):
    """Pairs of blocks, a half of the columns each; the bound is that of one block's columns (the slices are added in double)."""
    from test_gpu_prompt_routing import test_router_tiles as tiles
    tiles(F, E, H, T, normed)


@pytest.mark.parametrize("T", [75, 76, 200])   # 20 heads: 1,500 pairs, a block each; more: eight rows a warp
def test_prep_of_many_rows_in_both_forms(F, T):
    """Norm, rotation and append of a prompt's rows give the bits of the same rows in windows."""
    nq, nkv, ctx = 16, 2, 40
    g = torch.Generator(device="cuda").manual_seed(11)
    rnd = lambda *s: torch.randn(s, device="cuda", generator=g)
    qg, k, v, qn, kn = rnd(T, nq, 512), rnd(T, nkv, 256), rnd(T, nkv, 256), rnd(256), rnd(256)

    def run(step):
        q, kk = qg.clone(), k.clone()
        kc, vc = (torch.zeros((ctx + T, nkv, 256), dtype=torch.float16, device="cuda") for _ in range(2))
        for a in range(0, T, step):
            pos = torch.tensor([ctx + a], dtype=torch.int32, device="cuda")
            F.attn_prep_append(q[a:a + step], kk[a:a + step], v[a:a + step], qn, kn, kc, vc, pos)
        torch.cuda.synchronize()
        return q, kk, kc, vc
    for x, y in zip(run(T), run(32)):
        assert torch.equal(x, y)


def test_dense_of_no_rows(F):
    """No rows in, no rows out (nothing is launched)."""
    W = F.iq3s_retile(F.iq3s_quantize(torch.zeros(16 * 256, device="cuda")), 16, 256)
    y, err = F.dense(W, 16, 256, torch.empty((0, 256), device="cuda"))
    assert y.shape == (0, 16) and int(err.item()) == 0


def test_saving_a_sequence_that_is_not_there(F):
    cfg, e = _engine(F)
    try:
        for seq in (-1, cfg.n_seq):
            with pytest.raises(F.FnxError):
                e.save_state(seq)
    finally:
        e.close()


def test_lane_attention_far_into_a_cache(F):
    """Lanes whose sequences start some 2^26 rows into the caches (34 GB of keys): the same bits as at the front."""
    nq, nkv, stride, T = 8, 1, 1 << 20, 3
    rows = (64 + 2) * stride
    if torch.cuda.mem_get_info()[0] < 2.2 * rows * nkv * 512:
        pytest.skip("needs 70 GB")
    g = torch.Generator(device="cuda").manual_seed(5)
    kc, vc = (torch.empty((rows, nkv, 256), dtype=torch.float16, device="cuda") for _ in range(2))
    ctx = 200
    for t in (kc, vc):
        t[:ctx + T].normal_(0.0, 1.0, generator=g)
        for s in (63, 64, 65):
            t[s * stride:s * stride + ctx + T] = t[:ctx + T]
    qg = torch.randn((T, nq, 512), device="cuda", generator=g)
    L = F.lib()
    scratch = torch.empty(L.fnx_attn_scratch_bytes(T, nq, 256), dtype=torch.uint8, device="cuda")
    pos = torch.full((66,), ctx, dtype=torch.int32, device="cuda")
    row0 = torch.tensor([0, T], dtype=torch.int32, device="cuda")
    outs = []
    for s in (0, 63, 64, 65):
        out = torch.empty((T, nq, 256), device="cuda")
        lane = torch.tensor([s], dtype=torch.int32, device="cuda")
        F.check(L.fnx_attn_lanes(F.ptr(qg), nq * 512, F.ptr(kc), F.ptr(vc), stride, F.ptr(out), T, 1, nq, nkv, 256, F.ptr(pos), F.ptr(lane), F.ptr(row0), F.ptr(scratch), None))
        torch.cuda.synchronize()
        outs.append(out)
    assert all(torch.equal(o, outs[0]) for o in outs[1:])


@pytest.mark.parametrize("what", ["attention", "one KV head", "DeltaNet prompt"])
def test_scratch_on_an_eight_byte_boundary(F, what):
    """Scratch of exactly the size that the library asks for, eight bytes off a 16-byte boundary: the same bits as on one, and nothing written
    around it."""
    g = torch.Generator(device="cuda").manual_seed(6)
    rnd = lambda *s: torch.randn(s, device="cuda", generator=g)
    L = F.lib()
    if what == "DeltaNet prompt":
        nk, nv, hs, NS, T = 2, 4, 128, 4, 20        # (back to the slot it starts from: the history's copy takes the end of the scratch)
        ch = (2 * nk + nv) * hs
        x, ab, hist, S = rnd(T, ch + nv * hs), rnd(T, 2 * nv), rnd(NS, 3, ch), 0.1 * rnd(NS, nv, hs, hs)
        convw, dt, a, nw = rnd(ch, 4), rnd(nv), -rnd(nv).abs(), rnd(hs)
        need = L.fnx_gdn_prompt_scratch_bytes(T, nk, nv, hs)

        def run(at):
            y = torch.empty((T, nv * hs), device="cuda")
            h, s = hist.clone(), S.clone()
            F.check(L.fnx_gdn_prompt(F.ptr(x), x.stride(0), F.ptr(ab), ab.stride(0), F.ptr(h), F.ptr(convw), F.ptr(dt), F.ptr(a), F.ptr(nw), F.ptr(s), 1, NS, F.ptr(y), nk,
                                     nv, hs, T, 1e-6, C.c_void_p(at), None))
            return torch.cat([y.flatten(), h.flatten(), s.flatten()])
    else:
        nq, nkv, T, ctx = (16, 2, 5, 700) if what == "attention" else (8, 1, 9, 9600)
        qg, kc, vc = rnd(T, nq, 512), rnd(ctx + T, nkv, 256).half(), rnd(ctx + T, nkv, 256).half()
        pos = torch.tensor([ctx], dtype=torch.int32, device="cuda")
        need = L.fnx_attn_scratch_bytes(T, nq, 256)

        def run(at):
            out = torch.empty((T, nq, 256), device="cuda")
            F.check(L.fnx_attn(F.ptr(qg), nq * 512, F.ptr(kc), F.ptr(vc), F.ptr(out), T, nq, nkv, 256, F.ptr(pos), None, C.c_void_p(at), None))
            return out
    mem = torch.full((need + 4096,), 0x5A, dtype=torch.uint8, device="cuda")
    outs = []
    torch.cuda.synchronize()
    for off in (1024, 1032):
        mem.fill_(0x5A)
        torch.cuda.synchronize()
        outs.append(run(mem.data_ptr() + off))
        torch.cuda.synchronize()
        assert int((mem[:off] != 0x5A).sum()) == 0 and int((mem[off + need:] != 0x5A).sum()) == 0
    assert torch.equal(outs[0], outs[1])


def test_parking_where_no_thread_can_be_started(F, tmp_path):
    """pthread_create refused by a shim during save and load: the calling thread moves everything itself."""
    import os
    import pathlib
    import subprocess
    import sys
    (tmp_path / "shim.c").write_text("""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
static int refuse, refused;
void shim_refuse(int on) { refuse = on; }
int shim_refused(void) { return refused; }
int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* x) {
    static int (*real)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
    if (!real) real = dlsym(RTLD_NEXT, "pthread_create");
    if (refuse) { ++refused; return EAGAIN; }
    return real(t, a, f, x);
}
""")
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(tmp_path / "shim.so"), str(tmp_path / "shim.c"), "-ldl"], check=True)
    code = """
import ctypes, sys
sys.path[:0] = [%r, %r]
import torch
import fnx_b200 as F
from test_gpu_engine_edges import _engine
cfg, e = _engine(F, n_seq=2)
e.prompt(list(range(150)))
want = bytes(e.save_state(0))
shim = ctypes.CDLL(None)
shim.shim_refuse(1)
image = e.save_state(0)
e.load_state(image, 1)
shim.shim_refuse(0)
assert bytes(image) == want and bytes(e.save_state(1)) == want and shim.shim_refused() > 0
e.close()
print("same", shim.shim_refused())
""" % (str(pathlib.Path(F.PACKAGE_DIR).parent), str(pathlib.Path(__file__).parent))
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, LD_PRELOAD=str(tmp_path / "shim.so")), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("same"), r.stderr[-2000:]


def test_the_kept_counts_of_a_lanes_commit_can_be_read(F):
    cfg, e = _engine(F, n_seq=3)
    try:
        e.verify_lanes_rows([2, 0, 1], [[1, 2, 3], [4], [5, 6]])
        e.commit_lanes([2, 0, 1], [2, 1, 2])
        e.error_bits()                               # (waits for the commit)
        assert e.tensor("buf.lane_keep", torch.int32)[:3].tolist() == [2, 1, 2]
    finally:
        e.close()
