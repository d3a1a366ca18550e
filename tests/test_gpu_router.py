"""Router: logits bit-identical to the reference CUDA kernel's summation order, top-k indices
bit-exact against the reference's CPU router (sequential order), ties, bias, refusals."""
import numpy as np
import pytest
import torch

from tests.parity import load_ref_lib

pytestmark = pytest.mark.gpu


class _Router:
    def __init__(self, dev, E):
        self.dev = dev
        self.scores = torch.zeros(3 * E, dtype=torch.float32, device=dev)
        self.ids = torch.zeros(16, dtype=torch.int16, device=dev)
        self.w = torch.zeros(16, dtype=torch.float32, device=dev)
        self.ws = torch.zeros(4, dtype=torch.int32, device=dev)

    def run(self, x, W, k, mode, scaling, normalize=True, bias=None, exact=True):
        from vic_b200 import kernels
        kernels.router_topk_ex(x, W, self.scores, bias, self.ids, self.w, k, mode, scaling, normalize, exact, self.ws)
        torch.cuda.synchronize()
        assert int(self.ws[0].item()) == 0
        E = W.shape[0]
        return (self.ids[:k].cpu().numpy().view(np.uint16).copy(), self.w[:k].cpu().numpy().copy(),
                self.scores[:E].cpu().numpy().copy())


def test_logits_bit_identical_to_reference_order(cuda_dev, oracle):
    from vic_b200 import kernels
    g = torch.Generator(device="cpu").manual_seed(21)
    for E, H in [(8, 4096), (384, 7168), (5, 200)]:
        x = torch.randn(H, generator=g)
        W = torch.randn(E, H, generator=g) * 0.02
        W16 = W.to(torch.float16)
        scores = torch.zeros(E, dtype=torch.float32, device=cuda_dev)
        kernels.router_gemv_f32(x.to(cuda_dev), W16.to(cuda_dev), scores, H, E)
        want = oracle.router_logits(x.numpy(), W16.numpy(), oracle.ORDER_GPU128)
        assert np.array_equal(scores.cpu().numpy().view(np.uint32), want.view(np.uint32))
        ref = load_ref_lib()
        if ref is not None:
            theirs = torch.zeros(E, dtype=torch.float32, device=cuda_dev)
            xd, wd = x.to(cuda_dev), W16.to(cuda_dev)
            assert ref.vib3_launch_router_gemv_f32(xd.data_ptr(), wd.data_ptr(), theirs.data_ptr(), H, E,
                                                   torch.cuda.current_stream().cuda_stream) == 0
            torch.cuda.synchronize()
            assert np.array_equal(scores.cpu().numpy().view(np.uint32), theirs.cpu().numpy().view(np.uint32))
        # fp32 router weights, bf16 activations (the benchmark's configuration)
        r = _Router(cuda_dev, E)
        xb = x.to(torch.bfloat16)
        _, _, lg = r.run(xb.to(cuda_dev), W.to(cuda_dev), min(2, E), 1, 1.0, exact=False)
        want = oracle.router_logits(xb.float().numpy(), W.numpy(), oracle.ORDER_GPU128)
        assert np.array_equal(lg.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("name,E,H,k,mode,scaling,xdt,ntok", [
    ("mixtral", 8, 4096, 2, 0, 1.0, torch.float16, 3000),
    ("kimi", 384, 7168, 8, 1, 2.827, torch.bfloat16, 10000),
])
def test_topk_indices_bit_exact_vs_cpu_router(cuda_dev, oracle, name, E, H, k, mode, scaling, xdt, ntok):
    g = torch.Generator(device="cpu").manual_seed(1234)
    W = torch.randn(E, H, generator=g) * 0.02
    Wd = W.to(cuda_dev)
    Wn = W.numpy()
    r = _Router(cuda_dev, E)
    xs = torch.randn(ntok, H, generator=g).to(xdt)
    xs_d = xs.to(cuda_dev)
    xs_n = xs.float().numpy()
    mismatches_same_order = 0
    max_w_rel = 0.0
    for t in range(ntok):
        ids, w, _ = r.run(xs_d[t], Wd, k, mode, scaling, exact=True)
        oi, ow, _ = oracle.router(xs_n[t], Wn, k, mode, scaling, True, None, oracle.ORDER_SEQUENTIAL)
        assert np.array_equal(ids, oi), f"{name} token {t}: {ids} vs {oi}"
        max_w_rel = max(max_w_rel, float(np.max(np.abs(w - ow) / np.abs(ow))))
        if t < 500:
            ids2, _, _ = r.run(xs_d[t], Wd, k, mode, scaling, exact=False)
            oi2, _, _ = oracle.router(xs_n[t], Wn, k, mode, scaling, True, None, oracle.ORDER_GPU128)
            mismatches_same_order += int(not np.array_equal(ids2, oi2))
    assert mismatches_same_order == 0
    # weights move with the summation order of the logits (~1e-5 absolute on a logit)
    assert max_w_rel < 1e-4


def test_ties_and_near_ties(cuda_dev, oracle):
    g = torch.Generator(device="cpu").manual_seed(9)
    E, H, k = 384, 7168, 8
    W = torch.randn(E, H, generator=g) * 0.02
    x = torch.randn(H, generator=g).to(torch.bfloat16)
    base = oracle.router_logits(x.float().numpy(), W.numpy(), oracle.ORDER_SEQUENTIAL)
    top = np.argsort(-base)[:k]
    # exact ties: duplicate the rows of the best three experts into higher and lower indices
    W[300] = W[top[0]]
    W[2] = W[top[1]]
    # near ties: the same row with its columns summed in another order (a permutation of x and w together
    # is not available to the router, so instead nudge one weight by one ulp-scale amount)
    W[77] = W[top[2]]
    W[77, 5] += 1e-9
    r = _Router(cuda_dev, E)
    for mode, scaling in [(1, 2.827), (0, 1.0)]:
        ids, w, _ = r.run(x.to(cuda_dev), W.to(cuda_dev), k, mode, scaling, exact=True)
        oi, ow, _ = oracle.router(x.float().numpy(), W.numpy(), k, mode, scaling, True, None, oracle.ORDER_SEQUENTIAL)
        assert np.array_equal(ids, oi)
        assert np.allclose(w, ow, rtol=1e-4)
    # all-equal rows: lowest indices win in order
    W2 = W[:1].repeat(16, 1)
    ids, w, _ = _Router(cuda_dev, 16).run(x.to(cuda_dev), W2.to(cuda_dev), 4, 1, 1.0)
    assert ids.tolist() == [0, 1, 2, 3]


def test_selection_bias_and_flags(cuda_dev, oracle):
    g = torch.Generator(device="cpu").manual_seed(4)
    E, H, k = 384, 7168, 8
    W = torch.randn(E, H, generator=g) * 0.02
    bias = (torch.randn(E, generator=g) * 0.1).float()
    r = _Router(cuda_dev, E)
    for t in range(50):
        x = torch.randn(H, generator=g).to(torch.bfloat16)
        for normalize in (True, False):
            ids, w, _ = r.run(x.to(cuda_dev), W.to(cuda_dev), k, 1, 2.827, normalize, bias.to(cuda_dev))
            oi, ow, _ = oracle.router(x.float().numpy(), W.numpy(), k, 1, 2.827, normalize, bias.numpy(), oracle.ORDER_SEQUENTIAL)
            assert np.array_equal(ids, oi)
            assert np.allclose(w, ow, rtol=1e-4)


def test_reference_signature_topk(cuda_dev, oracle):
    """vib3_launch_router_topk with the reference's signature; for E=8 also against the reference's own kernel."""
    from vic_b200 import kernels
    g = torch.Generator(device="cpu").manual_seed(77)
    ref = load_ref_lib()
    for E, H, k, mode, scaling in [(8, 4096, 2, 0, 1.0), (384, 7168, 8, 1, 2.827), (256, 2048, 8, 1, 1.0)]:
        W16 = (torch.randn(E, H, generator=g) * 0.02).to(torch.float16)
        x = torch.randn(H, generator=g)
        scores = torch.zeros(E, dtype=torch.float32, device=cuda_dev)
        ids = torch.zeros(16, dtype=torch.int16, device=cuda_dev)
        ws = torch.zeros(16, dtype=torch.float32, device=cuda_dev)
        act = kernels.run_router_gpu_topk(x.to(cuda_dev), W16.to(cuda_dev), scores, None, ids, ws, H, E, k, mode, scaling)
        oi, ow, _ = oracle.router(x.numpy(), W16.numpy(), k, mode, scaling, True, None, oracle.ORDER_GPU128)
        assert [e for e, _ in act] == oi.tolist()
        assert np.allclose([w for _, w in act], ow, rtol=1e-4)
        if ref is not None and (E & (E - 1)) == 0:
            xd, wd = x.to(cuda_dev), W16.to(cuda_dev)
            s2 = torch.zeros(E, dtype=torch.float32, device=cuda_dev)
            i2 = torch.zeros(16, dtype=torch.int16, device=cuda_dev)
            w2 = torch.zeros(16, dtype=torch.float32, device=cuda_dev)
            assert ref.vib3_launch_router_topk(xd.data_ptr(), wd.data_ptr(), s2.data_ptr(), None, i2.data_ptr(), w2.data_ptr(),
                                               H, E, k, mode, scaling, torch.cuda.current_stream().cuda_stream) == 0
            torch.cuda.synchronize()
            assert i2[:k].cpu().numpy().view(np.uint16).tolist() == [e for e, _ in act]
            assert np.allclose(w2[:k].cpu().numpy(), [w for _, w in act], rtol=2e-4)


def test_router_refusals(cuda_dev):
    from vic_b200.lib import lib
    L = lib()
    t = torch.zeros(4096, dtype=torch.float32, device=cuda_dev)
    p = t.data_ptr()
    assert L.vib3_launch_router_topk(p, p, p, None, p, p, 64, 8, 9, 0, 1.0, None) == -2      # top_k > E
    assert L.vib3_launch_router_topk(p, p, p, None, p, p, 64, 8, 0, 0, 1.0, None) == -2
    assert L.vib3_launch_router_topk(p, p, p, None, p, p, 4, 513, 2, 0, 1.0, None) == -2    # > MAX_EXPERTS
    assert L.vib3_launch_router_topk(p, p, p, None, p, p, 64, 8, 17, 0, 1.0, None) == -2    # > MAX_ACTIVE_EXPERTS
    assert L.vib3_launch_router_topk(None, p, p, None, p, p, 64, 8, 2, 0, 1.0, None) == -3
    assert L.vib3_launch_router_topk(p, p, p, None, p, p, 64, 8, 2, 2, 1.0, None) == -1     # unknown scoring mode
    assert L.vib3_launch_router_topk_ex(p, 0, p, 1, p, None, None, p, p, 64, 8, 2, 0, 1.0, 1, 1, None, None) == -3  # no workspace
    assert L.vib3_launch_router_topk_ex(p, 5, p, 1, p, None, None, p, p, 64, 8, 2, 0, 1.0, 1, 1, p, None) == -1
    torch.cuda.synchronize()


@pytest.mark.parametrize("case", ["outlier", "offset", "fp16w_heavy_tail"])
def test_exact_order_bound_under_stress(cuda_dev, oracle, case):
    """The near-tie detector rests on a statistical bound on the difference between two fp32 summation orders.
    Inputs that stretch it: one activation of magnitude ~100 among N(0,1) values; router rows and activations
    with a large common offset (every logit carries the same big term); fp16 router weights with heavy-tailed
    activations.  3,400 tokens each, all through the batched launch; indices must equal the CPU router's
    (sequential order) for every token."""
    from vic_b200 import kernels
    E, H, k, T = 384, 7168, 8, 3400
    g = torch.Generator(device="cpu").manual_seed({"outlier": 5, "offset": 6, "fp16w_heavy_tail": 7}[case])
    W = torch.randn(E, H, generator=g) * 0.02
    x = torch.randn(T, H, generator=g)
    if case == "outlier":
        pos = torch.randint(0, H, (T,), generator=g)
        x[torch.arange(T), pos] = 100.0 * torch.sign(torch.randn(T, generator=g))
        xdt, W_used = torch.bfloat16, W
    elif case == "offset":
        W = W + 0.05
        x = x + 0.5
        xdt, W_used = torch.float32, W
    else:
        x = x / torch.sqrt(torch.rand(T, H, generator=g).clamp_(min=0.02))   # heavy tails
        xdt, W_used = torch.bfloat16, W.to(torch.float16)
    xs = x.to(xdt).to(cuda_dev)
    Wd = W_used.to(cuda_dev)
    ids = torch.zeros(T, 16, dtype=torch.int16, device=cuda_dev)
    ws = torch.zeros(T, 16, dtype=torch.float32, device=cuda_dev)
    scores = torch.zeros(128, 3 * E, dtype=torch.float32, device=cuda_dev)
    wk = torch.zeros(128, 4, dtype=torch.int32, device=cuda_dev)
    for t0 in range(0, T, 128):
        n = min(128, T - t0)
        kernels.router_topk_batch(xs[t0:t0 + n], Wd, scores, None, None, ids[t0:t0 + n], ws[t0:t0 + n], k, 1, 2.827, True, True, wk)
    torch.cuda.synchronize()
    assert int(wk[:, 0].abs().sum().item()) == 0 and int(wk[:, 2].abs().sum().item()) == 0
    ids_n = ids[:, :k].cpu().numpy().view(np.uint16)
    ws_n = ws[:, :k].cpu().numpy()
    xs_n = xs.float().cpu().numpy()
    W_n = W_used.numpy()
    bad = 0
    for t in range(T):
        oi, ow, _ = oracle.router(xs_n[t], W_n, k, 1, 2.827, True, None, oracle.ORDER_SEQUENTIAL)
        if not np.array_equal(ids_n[t], oi):
            bad += 1
        else:
            assert np.allclose(ws_n[t], ow, rtol=2e-4), t
    assert bad == 0, f"{bad} of {T} tokens selected other experts than the CPU router ({case})"
    assert int(wk[:, 1].sum().item()) > 0 or case == "offset"   # the recomputation path was taken at least once


@pytest.mark.parametrize("E,H,ntok,xdt,wdt", [
    (5, 264, 9, torch.bfloat16, torch.float32), (3, 128, 12, torch.float16, torch.float16), (384, 1024, 13, torch.float32, torch.float32),
    (7, 2056, 48, torch.bfloat16, torch.float16), (64, 520, 49, torch.float16, torch.float32), (16, 7168, 128, torch.bfloat16, torch.float32),
    (384, 264, 10, torch.bfloat16, torch.float32), (384, 264, 10, torch.float32, torch.float16), (340, 256, 12, torch.float16, torch.float16)])
def test_batched_logits_equal_single_token_logits(cuda_dev, E, H, ntok, xdt, wdt):
    """Token counts around the widths of the batched kernel, expert counts that leave rows of a CTA empty or few SMs to a second
    CTA of the same rows, row lengths that leave lanes without an item: every logit is the single-token launch's bit for bit."""
    from vic_b200 import kernels
    g = torch.Generator(device=cuda_dev).manual_seed(E * H + ntok)
    W = (0.05 * torch.randn(E, H, generator=g, device=cuda_dev)).to(wdt)
    xs = torch.randn(ntok, H, generator=g, device=cuda_dev).to(xdt)
    k = min(3, E)
    def buffers(n):
        return (torch.zeros(n, 3 * E, device=cuda_dev), torch.zeros(n, 16, dtype=torch.int16, device=cuda_dev),
                torch.zeros(n, 16, device=cuda_dev), torch.zeros(n, 4, dtype=torch.int32, device=cuda_dev))
    sc, ids, wt, ws = buffers(ntok)
    kernels.router_topk_batch(xs, W, sc, None, None, ids, wt, k, 1, 2.5, True, 0, ws)
    for t in range(ntok):
        s1, i1, w1, ws1 = buffers(1)
        kernels.router_topk_batch(xs[t:t + 1], W, s1, None, None, i1, w1, k, 1, 2.5, True, 0, ws1)
        torch.cuda.synchronize()
        assert torch.equal(sc[t, :E], s1[0, :E]) and torch.equal(ids[t], i1[0]) and torch.equal(wt[t], w1[0]), t


@pytest.mark.parametrize("H,offset", [(268, 0), (7172, 0), (520, 4), (268, 4)])
def test_rows_that_a_bulk_copy_cannot_take(cuda_dev, oracle, H, offset):
    """fp16 router rows that are not whole 16-byte units, or that start on an 8-byte boundary only, with fp32 tokens: they
    belong to the direct kernel, for one token and for a batch."""
    from vic_b200 import kernels
    E, T, k = 7, 11, 3
    g = torch.Generator(device="cpu").manual_seed(H + offset)
    W = (0.05 * torch.randn(E, H, generator=g)).to(torch.float16)
    Wd = torch.zeros(E * H + offset, dtype=torch.float16, device=cuda_dev)[offset:].view(E, H)
    Wd.copy_(W)
    assert Wd.data_ptr() % 16 == 2 * offset
    xs = torch.randn(T, H, generator=g)
    xs_d = xs.to(cuda_dev)
    want = [oracle.router_logits(xs[t].numpy(), W.numpy(), oracle.ORDER_GPU128) for t in range(T)]
    picks = [oracle.router(xs[t].numpy(), W.numpy(), k, 1, 2.5, True, None, oracle.ORDER_SEQUENTIAL)[0] for t in range(T)]
    for n in (1, 2, T):
        sc, ids = torch.zeros(n, 3 * E, device=cuda_dev), torch.zeros(n, 16, dtype=torch.int16, device=cuda_dev)
        wt, ws = torch.zeros(n, 16, device=cuda_dev), torch.zeros(n, 4, dtype=torch.int32, device=cuda_dev)
        kernels.router_topk_batch(xs_d[:n], Wd, sc, None, None, ids, wt, k, 1, 2.5, True, 0, ws)
        sc_n = sc[:, :E].cpu().numpy()
        assert all(np.array_equal(sc_n[t].view(np.uint32), want[t].view(np.uint32)) for t in range(n))
        kernels.router_topk_batch(xs_d[:n], Wd, sc, None, None, ids, wt, k, 1, 2.5, True, 1, ws)
        assert all(np.array_equal(ids[t, :k].cpu().numpy().view(np.uint16), picks[t]) for t in range(n))


@pytest.mark.parametrize("H,cands,T,xdt,wdt", [
    (264, 2, 2, torch.bfloat16, torch.float32), (520, 9, 9, torch.float32, torch.float32), (520, 17, 13, torch.float16, torch.float32),
    (776, 7, 13, torch.float32, torch.float16), (776, 8, 8, torch.bfloat16, torch.float16), (1016, 9, 2, torch.float16, torch.float16),
    (7168, 17, 9, torch.bfloat16, torch.float32)])
def test_batched_recomputation_of_near_ties(cuda_dev, oracle, H, cands, T, xdt, wdt):
    """Every other token has `cands` near-tied experts at the top: one trip of the recomputation or several, last blocks that are
    short, odd numbers of blocks.  The near-tied logits are then the CPU router's to the bit, all others the reference
    kernel's, the selection is the CPU router's, and only those tokens count a recomputation."""
    from vic_b200 import kernels
    E, k = 40, 3
    g = torch.Generator(device="cpu").manual_seed(H + cands)
    base = torch.randn(H, generator=g)
    W = torch.randn(E, H, generator=g) * (0.3 / H ** 0.5)
    tied = torch.randperm(E, generator=g)[:cands].sort().values
    W[tied] = 2 * base / base.dot(base)          # a logit of about 2; -2 for the other tokens
    if wdt == torch.float32:                     # near ties and not only equal rows: differences below the sums' rounding
        W[tied] *= 1 + 2.0 ** -22 * torch.randn(cands, H, generator=g)
    W = W.to(wdt)
    sign = torch.where(torch.arange(T) % 2 == 0, 1.0, -1.0)
    xs = (sign[:, None] * base + 0.1 * torch.randn(T, H, generator=g)).to(xdt)
    xs_n, W_n = xs.float().numpy(), W.numpy()

    def run(x):
        n = x.shape[0]
        sc, ids = torch.zeros(n, 3 * E, device=cuda_dev), torch.zeros(n, 16, dtype=torch.int16, device=cuda_dev)
        wt, ws = torch.zeros(n, 16, device=cuda_dev), torch.zeros(n, 4, dtype=torch.int32, device=cuda_dev)
        kernels.router_topk_batch(x, Wd, sc, None, None, ids, wt, k, 1, 2.5, True, 1, ws)
        return sc.cpu().numpy(), ids[:, :k].cpu().numpy().view(np.uint16), wt[:, :k].cpu().numpy(), ws.cpu().numpy()

    Wd, xs_d = W.to(cuda_dev), xs.to(cuda_dev)
    sc, ids, wt, ws = run(xs_d)
    assert ws[:, 1].tolist() == [1 if t % 2 == 0 else 0 for t in range(T)] and not ws[:, [0, 2, 3]].any()
    for t in range(T):
        want = oracle.router_logits(xs_n[t], W_n, oracle.ORDER_GPU128)
        if t % 2 == 0:
            want[tied.numpy()] = oracle.router_logits(xs_n[t], W_n, oracle.ORDER_SEQUENTIAL)[tied.numpy()]
        assert np.array_equal(sc[t, :E].view(np.uint32), want.view(np.uint32)), t
        oi, ow, _ = oracle.router(xs_n[t], W_n, k, 1, 2.5, True, None, oracle.ORDER_SEQUENTIAL)
        assert np.array_equal(ids[t], oi), t
        assert np.allclose(wt[t], ow, rtol=2e-4), t
        # sums of |x w|: a chain of at most H / 64 roundings and a tree of at most 8, in both forms
        one = run(xs_d[t:t + 1])[0][0]
        assert np.allclose(sc[t, E:2 * E], one[E:2 * E], rtol=(H / 64 + 8) * 2.0 ** -23, atol=0), t
