"""Each kernel alone against its plain reference, at sizes other than the models'."""
import ctypes
import math

import numpy as np
import pytest
import torch

import plain_qwen3 as P

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DTYPES = [torch.float32, torch.bfloat16]


def ops():
    from velox_b200.csrc import ops as o
    return o


def close(got, want, dtype, atol32=2e-5, what=""):
    """A kernel against the plain operation on the SAME inputs (already rounded to the
    kernel's element type).  float32: atol32 + 1e-5 |x|.  bfloat16: all that separates the
    two is the rounding of the result (and, in attention, of the probabilities) to
    bfloat16, 2^-9 relative each: a value may be off by 2^-7 of the largest value of its
    row, plus 2^-10 for rows near zero."""
    got = got.detach().double().cpu().numpy()
    want = np.asarray(want, np.float64)
    assert got.shape == want.shape, (got.shape, want.shape)
    assert np.isfinite(got).all(), what + ": non-finite output"
    err = np.abs(got - want)
    if dtype == torch.float32:
        bound = atol32 + 1e-5 * np.abs(want)
    else:
        flat = np.abs(want).reshape(-1, want.shape[-1])
        bound = (2.0 ** -7 * flat.max(axis=1, keepdims=True) + 2.0 ** -10).reshape(want.shape[:-1] + (1,))
    assert (err <= bound).all(), "%s: max err %.3g at %s" % (what, err.max(), np.unravel_index((err - bound).argmax(), err.shape))


def rnd(shape, dtype, seed, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(shape, generator=g) * scale).to(dtype).to(DEV)


def f64(t):
    return t.detach().double().cpu().numpy()


# ----------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", DTYPES)
def test_embedding(dtype):
    table = rnd((37, 50), dtype, 0)
    ids = torch.tensor([0, 36, 5, 5, 17], dtype=torch.int32, device=DEV)
    out = ops().embedding(ids, table)
    assert out.dtype == torch.float32
    assert torch.equal(out, table.float()[ids.long()])
    bad = ops().embedding(torch.tensor([3, 37], dtype=torch.int32, device=DEV), table)
    assert torch.isnan(bad[1]).all() and torch.equal(bad[0], table.float()[3])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("width", [48, 1000, 4100])
def test_add_rmsnorm(dtype, width):
    rows, eps = 7, 1e-5
    res = rnd((rows, width), torch.float32, 1)
    delta = rnd((rows, width), dtype, 2)
    w = (1 + 0.05 * torch.randn(width)).to(DEV)
    want_sum = f64(res) + f64(delta)
    want = P.rms_norm(want_sum, f64(w), eps)
    r = res.clone()
    out = ops().add_rmsnorm(r, delta, w, eps, dtype)
    close(out, want, dtype, what="normed")
    assert np.allclose(f64(r), want_sum, atol=1e-6)  # the residual holds the float32 sum
    # no delta: residual untouched
    r2 = res.clone()
    out2 = ops().add_rmsnorm(r2, None, w, eps, dtype)
    close(out2, P.rms_norm(f64(res), f64(w), eps), dtype)
    assert torch.equal(r2, res)
    # gathered rows: only those are normed, the residual stays
    idx = torch.tensor([6, 0, 3], dtype=torch.int32, device=DEV)
    r3 = res.clone()
    out3 = ops().add_rmsnorm(r3, delta, w, eps, dtype, rows=idx)
    close(out3, want[[6, 0, 3]], dtype)
    assert torch.equal(r3, res)


@pytest.mark.parametrize("dtype", DTYPES)
def test_rmsnorm_rows(dtype):
    x = rnd((11, 80), dtype, 3)
    w = (1 + 0.05 * torch.randn(80)).to(DEV)
    close(ops().rmsnorm(x, w, 1e-6), P.rms_norm(f64(x), f64(w), 1e-6), dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("act", ["silu", "gelu", "gelu_pytorch_tanh", "relu"])
def test_gated_act(dtype, act):
    x = rnd((9, 2 * 75), dtype, 4, 2.0)
    g, u = f64(x)[:, :75], f64(x)[:, 75:]
    if act == "silu":
        a = P.silu(g)
    elif act == "gelu":
        a = 0.5 * g * (1 + np.vectorize(math.erf)(g / math.sqrt(2)))
    elif act == "gelu_pytorch_tanh":
        a = 0.5 * g * (1 + np.tanh(math.sqrt(2 / math.pi) * (g + 0.044715 * g ** 3)))
    else:
        a = np.maximum(g, 0)
    close(ops().gated_act(x, act), a * u, dtype)
    # the same values laid out in tiles of 5 gates followed by their 5 ups
    tiled = torch.stack([x[:, :75].reshape(9, 15, 5), x[:, 75:].reshape(9, 15, 5)], 2).reshape(9, 150).contiguous()
    assert torch.equal(ops().gated_act(tiled, act, block=5), ops().gated_act(x, act))


# ----------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("H,Hk,D,rot,S", [(6, 3, 48, 48, 8), (5, 1, 16, 8, 4), (8, 2, 128, 128, 16), (2, 2, 80, 0, 2)])
def test_qk_norm_rope_kv(dtype, H, Hk, D, rot, S):
    T, pages, eps, theta = 13, 9, 1e-5, 1e6
    qkv = rnd((T, (H + 2 * Hk) * D), dtype, 5)
    qw = (1 + 0.05 * torch.randn(D)).to(DEV)
    kw = (1 + 0.05 * torch.randn(D)).to(DEV)
    positions = torch.tensor([0, 1, 2, 77, 78, 5000, 5001, 31, 32, 33, 3, 40000, 9], dtype=torch.int32, device=DEV)
    slots = torch.randperm(pages * S)[:T].to(torch.int32).to(DEV)
    k_pool = torch.full((pages, Hk, S, D), float("nan"), dtype=dtype, device=DEV)
    v_pool = torch.full((pages, Hk, S, D), float("nan"), dtype=dtype, device=DEV)
    inv = None
    if rot:
        inv = torch.tensor([np.float32(1.0) / np.float32(theta ** (i / rot)) for i in range(0, rot, 2)],
                           dtype=torch.float32, device=DEV)
    x = f64(qkv)
    q = x[:, : H * D].reshape(T, H, D)
    k = x[:, H * D : (H + Hk) * D].reshape(T, Hk, D)
    v = x[:, (H + Hk) * D :].reshape(T, Hk, D)
    qn, kn = P.rms_norm(q, f64(qw), eps), P.rms_norm(k, f64(kw), eps)
    if rot:
        pos = positions.cpu().numpy()
        qn = np.concatenate([P.rope(qn[..., :rot], pos, theta), qn[..., rot:]], -1)
        kn = np.concatenate([P.rope(kn[..., :rot], pos, theta), kn[..., rot:]], -1)
    work = qkv.clone()
    ops().qk_norm_rope_kv(work, qw, kw, eps, inv, rot, positions, slots, k_pool, v_pool, H, Hk, D)
    close(work[:, : H * D].reshape(T, H, D), qn, dtype, what="q")
    sl = slots.cpu().numpy()
    got_k = k_pool[sl // S, :, sl % S, :]
    got_v = v_pool[sl // S, :, sl % S, :]
    close(got_k, kn, dtype, what="k in the pool")
    assert torch.equal(got_v, qkv[:, (H + Hk) * D :].reshape(T, Hk, D))  # values are copied bit for bit
    untouched = torch.ones(pages * S, dtype=torch.bool)
    untouched[sl] = False
    assert torch.isnan(k_pool.reshape(pages, Hk, S, D).permute(0, 2, 1, 3).reshape(pages * S, -1)[untouched]).all()
    # without a slot mapping nothing is written and keys are treated in place
    work2 = qkv.clone()
    ops().qk_norm_rope_kv(work2, qw, kw, eps, inv, rot, positions, None, None, None, H, Hk, D)
    close(work2[:, H * D : (H + Hk) * D].reshape(T, Hk, D), kn, dtype, what="k in place")
    assert torch.equal(work2[:, (H + Hk) * D :], qkv[:, (H + Hk) * D :])


def test_qk_norm_rope_kv_for_many_tokens_gives_the_same_bits():
    """From 64 tokens on the bfloat16 kernel for heads of 128 works row by row with the
    token's cosines and sines shared by all heads; the result is the one of the
    kernel for few tokens, bit for bit."""
    H, Hk, D, S, T, pages, eps = 6, 2, 128, 16, 150, 12, 1e-6
    qkv = rnd((T, (H + 2 * Hk) * D), torch.bfloat16, 6, 2.0)
    qw, kw = (1 + 0.05 * torch.randn(D)).to(DEV), (1 + 0.05 * torch.randn(D)).to(DEV)
    positions = torch.randint(0, 40000, (T,), dtype=torch.int32).to(DEV)
    slots = torch.randperm(pages * S)[:T].to(torch.int32)
    slots[17] = -1                                            # a row that writes nothing
    slots = slots.to(DEV)
    inv = torch.from_numpy(P.rope_inverse_frequencies(D, 1e6)).to(DEV)
    outs = []
    for step in (T, 50):                                      # all at once; in slices below 64 tokens
        work = qkv.clone()
        kp = torch.full((pages, Hk, S, D), float("nan"), dtype=torch.bfloat16, device=DEV)
        vp = torch.full_like(kp, float("nan"))
        for a in range(0, T, step):
            part = work[a:a + step].contiguous()
            ops().qk_norm_rope_kv(part, qw, kw, eps, inv, D, positions[a:a + step].contiguous(),
                                  slots[a:a + step].contiguous(), kp, vp, H, Hk, D)
            work[a:a + step] = part
        outs.append((work, kp, vp))
    for x, y in zip(*outs):
        assert torch.equal(torch.nan_to_num(x.float(), nan=-7.0), torch.nan_to_num(y.float(), nan=-7.0))
    assert int(torch.isnan(outs[0][1].float()).sum()) == (pages * S - (T - 1)) * Hk * D


# ----------------------------------------------------------------------------
def paged_case(dtype, seqs, H, Hk, D, S, window, seed, spike=None):
    """seqs: list of (kv_offset, new_tokens).  Builds whole sequences, scatters
    keys/values into scattered pages, and returns kernel inputs + the plain answer."""
    rng = np.random.default_rng(seed)
    total_pages = sum(-(-(o + n) // S) for o, n in seqs) + 5
    perm = rng.permutation(total_pages)
    k_pool = torch.full((total_pages, Hk, S, D), float("nan"), dtype=dtype, device=DEV)
    v_pool = torch.full((total_pages, Hk, S, D), float("nan"), dtype=dtype, device=DEV)
    max_blocks = max(-(-(o + n) // S) for o, n in seqs) + 2
    bt = np.full((len(seqs), max_blocks), -1, np.int32)
    qs, pos, sot, want = [], [], [], []
    used = 0
    for i, (off, n) in enumerate(seqs):
        L = off + n
        q = torch.randn(L, H, D, generator=torch.Generator().manual_seed(seed * 100 + i)).to(dtype)
        k = torch.randn(L, Hk, D, generator=torch.Generator().manual_seed(seed * 100 + 50 + i)).to(dtype)
        v = torch.randn(L, Hk, D, generator=torch.Generator().manual_seed(seed * 100 + 70 + i)).to(dtype)
        if spike is not None and L > spike:
            # one far key that every late query of head 0 must find: its score
            # towers over the others, so the output is that key's value
            j = spike
            q[-1, 0] = 0; q[-1, 0, 0] = 12.0
            k[j, 0] = 0; k[j, 0, 0] = 12.0
        npg = -(-L // S)
        pages = perm[used:used + npg]
        used += npg
        bt[i, :npg] = pages
        for p in range(L):
            k_pool[pages[p // S], :, p % S] = k[p].to(DEV)
            v_pool[pages[p // S], :, p % S] = v[p].to(DEV)
        ref = P.causal_attention(f64(q), f64(k), f64(v), window)
        qs.append(q[off:])
        want.append(ref[off:])
        pos += list(range(off, L))
        sot += [i] * n
    q_all = torch.cat(qs).reshape(-1, H * D).contiguous().to(DEV)
    return (q_all, k_pool, v_pool, torch.from_numpy(bt).to(DEV), torch.tensor(sot, dtype=torch.int32, device=DEV),
            torch.tensor(pos, dtype=torch.int32, device=DEV), np.concatenate(want).reshape(-1, H * D))


ATT_CASES = [
    # (seqs, H, Hk, D, S, window)
    ([(0, 1)], 4, 2, 16, 4, 0),                              # a sequence's first token
    ([(0, 3), (0, 2), (0, 1)], 4, 4, 32, 8, 0),              # first tokens, no grouping
    ([(0, 8), (20, 4), (10, 1)], 8, 2, 64, 4, 0),            # the reference's mixed batch: cold 8, warm 4 @20, decode 1 @10
    ([(239, 1)] * 8, 8, 2, 128, 16, 0),                      # 8 decodes over 240 keys
    ([(0, 37)], 6, 3, 48, 8, 0),                             # head size 48, 3 groups, a partial last page
    ([(0, 50), (45, 5), (63, 1)], 4, 1, 80, 16, 13),         # a window that is no multiple of the page
    ([(300, 2)], 2, 1, 256, 16, 0),                          # the largest head size
    ([(31, 1), (32, 1), (33, 1)], 4, 2, 16, 16, 0),          # around a page's edge
    ([(0, 21), (40, 3)], 6, 2, 40, 4, 0),                    # a head size that is even and no multiple of 16
]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("case", range(len(ATT_CASES)))
def test_paged_attention_generic(dtype, case):
    seqs, H, Hk, D, S, window = ATT_CASES[case]
    q, kp, vp, bt, sot, pos, want = paged_case(dtype, seqs, H, Hk, D, S, window, seed=case)
    out = ops().paged_attention_generic(q, H * D, kp, vp, bt, sot, pos, 1 / math.sqrt(D), window, H, Hk, D, q.shape[0])
    close(out, want, dtype, atol32=1e-5, what="attention case %d" % case)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("far", [0, 3, 250, 511])
def test_attention_finds_one_far_key_among_hundreds(dtype, far):
    H, Hk, D, S = 4, 2, 64, 16
    q, kp, vp, bt, sot, pos, want = paged_case(dtype, [(599, 1)], H, Hk, D, S, 0, seed=11, spike=far)
    out = ops().paged_attention_generic(q, H * D, kp, vp, bt, sot, pos, 1 / math.sqrt(D), 0, H, Hk, D, 1)
    close(out, want, dtype, atol32=1e-5)
    # the spike dominates: head 0's output is (nearly) the far key's value
    page, off = int(bt[0, far // S]), far % S
    assert torch.allclose(out[0, :D].float(), vp[page, 0, off].float(), atol=5e-2)


@pytest.mark.parametrize("H,Hk,D,Dv", [(4, 2, 128, 128), (3, 3, 64, 128), (10, 2, 36, 20), (8, 1, 128, 64)])
def test_float32_attention_whatever_tokens_a_block_has(H, Hk, D, Dv):
    """The 32-bit path of layers without a window: blocks of up to eight neighbouring tokens, whole rounds of 128 keys and remainders; with a
    soft cap, a bias by distance, sinks and a gate.  Against the kernel that a window beyond all keys selects, whose sums have another
    order (the tolerance of `close`), and every token alone bit for bit; what no token sees may be anything."""
    S, lens = 16, [(1, 0), (1, 127), (1, 400), (13, 250), (40, 3), (9, 1000)]     # (new tokens, cached)
    need = [-(-(n + c) // S) for n, c in lens]
    bt = torch.zeros((len(lens), max(need)), dtype=torch.int32)
    order, at = torch.randperm(sum(need), generator=torch.Generator().manual_seed(0)).to(torch.int32), 0
    for i, n in enumerate(need):
        bt[i, :n], at = order[at:at + n], at + n
    k, v = rnd((sum(need), Hk, S, D), torch.float32, 1), rnd((sum(need), Hk, S, Dv), torch.float32, 2)
    for i, (n, c) in enumerate(lens):     # what lies behind a request's last key
        if (n + c) % S:
            page = int(bt[i, need[i] - 1])
            v[page, :, (n + c) % S:] = float("nan")
            k[page, :, (n + c) % S:] = float("inf")
    bt = bt.to(DEV)
    seq = torch.tensor([i for i, (n, c) in enumerate(lens) for _ in range(n)], dtype=torch.int32, device=DEV)
    pos = torch.tensor([c + j for n, c in lens for j in range(n)], dtype=torch.int32, device=DEV)
    T = len(pos)
    q = rnd((T, H * D + H), torch.float32, 3)
    more = dict(v_head_dim=Dv, softcap=20.0, bias_exponent=8.0, sinks=rnd((H,), torch.float32, 4), gate_col=H * D)

    def run(q, seq, pos, window, **kw):
        return ops().paged_attention_generic(q, q.shape[1], k, v, bt, seq, pos, D ** -0.5, window, H, Hk, D, len(pos), **kw)

    for kw in (dict(v_head_dim=Dv), more):
        whole = run(q, seq, pos, 0, **kw)
        close(whole, f64(run(q, seq, pos, 4096, **kw)), torch.float32)
        for t in range(T):
            assert torch.equal(run(q[t:t + 1], seq[t:t + 1], pos[t:t + 1], 0, **kw)[0], whole[t]), t


@pytest.mark.parametrize("H,Hk,D,Dv", [(16, 16, 128, 128), (16, 8, 64, 128), (8, 2, 96, 36), (12, 12, 36, 20)])
def test_float32_attention_of_many_decoded_tokens(H, Hk, D, Dv):
    """So many requests with a token each that their blocks would take turns: the form without sharing, with the bits that the shared one gives a few
    of them, with a soft cap, a bias by distance, sinks and a gate as well."""
    S, lens = 16, [1 + 37 * i % 611 for i in range(90)]
    need = [-(-n // S) for n in lens]
    bt = torch.zeros((len(lens), max(need)), dtype=torch.int32)
    order, at = torch.randperm(sum(need), generator=torch.Generator().manual_seed(0)).to(torch.int32), 0
    for i, n in enumerate(need):
        bt[i, :n], at = order[at:at + n], at + n
    bt = bt.to(DEV)
    k, v = rnd((sum(need), Hk, S, D), torch.float32, 1), rnd((sum(need), Hk, S, Dv), torch.float32, 2)
    q = rnd((len(lens), H * D + H), torch.float32, 3)
    seq, pos = torch.arange(len(lens), dtype=torch.int32, device=DEV), torch.tensor([n - 1 for n in lens], dtype=torch.int32, device=DEV)

    def run(lo, hi, **kw):   # (the block table of the tokens' own requests: a call knows how many there are)
        return ops().paged_attention_generic(q[lo:hi], q.shape[1], k, v, bt[lo:hi], seq[lo:hi] - lo, pos[lo:hi], D ** -0.5, 0, H, Hk, D, hi - lo,
                                             v_head_dim=Dv, **kw)

    for kw in (dict(), dict(softcap=20.0, bias_exponent=8.0, sinks=rnd((H,), torch.float32, 4), gate_col=H * D)):
        whole = run(0, len(lens), **kw)
        for lo in range(0, len(lens), 6):
            assert torch.equal(run(lo, lo + 6, **kw), whole[lo:lo + 6]), lo


# ----------------------------------------------------------------------------
@pytest.mark.parametrize("M,N,K", [(1, 53, 71), (37, 64, 16), (130, 129, 100), (5, 384, 96)])
def test_gemm_simt_fp32(M, N, K):
    a, w = rnd((M, K), torch.float32, 6), rnd((N, K), torch.float32, 7)
    bias = rnd((N,), torch.float32, 8)
    close(ops().gemm_nt_simt(a, w), f64(a) @ f64(w).T, torch.float32)
    close(ops().gemm_nt_simt(a, w, bias), f64(a) @ f64(w).T + f64(bias), torch.float32)
    # a row's result does not depend on the rows beside it: bit-identical
    alone = ops().gemm_nt_simt(a[M - 1 :].contiguous(), w)
    assert torch.equal(alone[0], ops().gemm_nt_simt(a, w)[M - 1])


def float32_parts(K):
    """How the 32-bit product cuts k: (parts, their length)."""
    parts = min(8, max(1, K // (256 if K >= 1024 else 64)))
    length = -(-(-(-K // parts)) // 32) * 32
    return -(-K // length), length


@pytest.mark.parametrize("N,K,pad", [(64, 256, 0), (65, 512, 0), (130, 777, 0), (63, 1000, 3), (100, 2051, 1), (1024, 2048, 4), (40000, 300, 0),
                                     (8192, 128, 0), (8192, 256, 0), (8190, 512, 4), (8192, 1001, 0), (8192, 1024, 0)])
def test_gemm_float32_tiles_and_parts(N, K, pad):
    """The 32-bit product at the edges of its row tiles (4, 8, 16, 32, 64) and of the parts of k, rows that begin on 16-byte
    addresses and rows that do not, tiles enough to keep k whole and too few; every row the same bits however many rows the call has.
    A sum's error is at most (the additions that a term passes through) units of 2^-24 of the sum of the terms' sizes: half a
    part, the parts, two."""
    parts, length = float32_parts(K)
    steps = length // 2 + parts + 2
    w = rnd((N, K + pad), torch.float32, 7)[:, :K]
    a = rnd((130, K + pad), torch.float32, 6)[:, :K]
    bias = rnd((N,), torch.float32, 8)
    whole = ops().gemm_nt_simt(a, w, bias)
    limit = steps * 2.0 ** -24 * (abs(f64(a)) @ abs(f64(w)).T + abs(f64(bias)))
    assert (abs(f64(whole) - (f64(a) @ f64(w).T + f64(bias))) <= limit).all()
    for M in (1, 3, 4, 5, 8, 9, 16, 17, 32, 33, 63, 64, 65, 129):
        assert torch.equal(ops().gemm_nt_simt(a[130 - M:], w, bias), whole[130 - M:]), M


@pytest.mark.parametrize("K", [256, 512, 1000, 1024])
def test_gemm_float32_error_follows_the_parts(K):
    """Normal terms: a chain's j-th addition is rounded at the size of j^1/2 terms, so P parts of length L, two chains of L/2 each, come to an error
    of c 2^-24 (L/4 + 1 + (P + 1)/2)^1/2 of the result, c about 0.43 for roundings spread evenly: 0.6 allows for the draw.  (Two parts
    at k = 512 would come to 0.43 x 8.2 = 3.5 units, eight may have 0.6 x 4.6 = 2.8.)"""
    parts, length = float32_parts(K)
    a, w = rnd((64, K), torch.float32, 21), rnd((512, K), torch.float32, 22)
    want = f64(a) @ f64(w).T
    err = np.linalg.norm(f64(ops().gemm_nt_simt(a, w)) - want) / np.linalg.norm(want)
    assert err <= 0.6 * 2.0 ** -24 * math.sqrt(length / 4 + 1 + (parts + 1) / 2), err


@pytest.mark.parametrize("N,K,pad", [(1, 1024, 0), (127, 1056, 4), (129, 1025, 3), (1024, 2049, 3), (32768, 1032, 0), (256, 4096, 0),
                                     (6144, 1024, 0), (6144, 2560, 0), (4000, 1792, 0)])
def test_gemm_float32_by_three_parts(N, K, pad):
    """The 32-bit product on the tensor cores at the edges of its tiles (16, 32, 64, 128 rows, 128 columns), runs (32 k),
    chunks (64) and parts, which are dealt one, two or four to a block of a cluster or not at all (7 by twos leave one).  A term passes at most ten additions in its accumulator, each cut off below 2^-23 of the sum of the terms' sizes, the
    run's among those of its part and the part's, rounded to 2^-24; the products left out are below 3 x 2^-24."""
    assert ops()._f32_takes_tc(N, K)
    parts = min(8, max(1, K // 256))
    steps = 2 * 10 + -(-K // (32 * parts)) + 2 + parts + 3
    w = rnd((N, K + pad), torch.float32, 7)[:, :K]
    a = rnd((257, K + pad), torch.float32, 6)[:, :K]
    whole = ops().gemm_nt_simt(a, w)
    assert (abs(f64(whole) - f64(a) @ f64(w).T) <= steps * 2.0 ** -24 * (abs(f64(a)) @ abs(f64(w)).T)).all()
    for M in (1, 15, 16, 17, 31, 33, 64, 65, 127, 128, 129):
        assert torch.equal(ops().gemm_nt_simt(a[257 - M:], w), whole[257 - M:]), M


@pytest.mark.parametrize("K", [512, 1024, 2560])
def test_gemm_float32_infinities_nan_and_tiny_sums(K):
    """Infinities, NaN, sums that overflow and operands so small that their parts vanish in bfloat16: what multiply-adds give (at 512
    they form the product)."""
    a, w = rnd((5, K), torch.float32, 1), rnd((70, K), torch.float32, 2)
    a[1, 7], w[3, 9], w[4, 10], w[6], w[8] = math.inf, -math.inf, math.nan, 0.0, 1.0
    a[2] = 3e38
    a[3] *= 1e-20
    w[5] = w[5].abs() * 1e-16
    got = f64(ops().gemm_nt_simt(a, w))
    assert got[2, 8] == math.inf
    rows = [0, 1, 3, 4]
    got, A, W = got[rows], f64(a)[rows], f64(w)
    with np.errstate(invalid="ignore"):
        want, size = A @ W.T, abs(A) @ abs(W).T
    assert np.array_equal(np.isnan(got), np.isnan(want))     # (infinity times 0 in row 1, column 6; the NaN's column)
    infinite, finite = np.isinf(want), np.isfinite(want)
    assert infinite.any() and np.array_equal(got[infinite], want[infinite])
    assert (abs(got[finite] - want[finite]) <= (K * 2.0 ** -24 * size + K * 2.0 ** -149)[finite]).all()


def test_gemm_float32_takes_the_tensor_cores_where_few_rows_are_no_slower():
    """The choice by N and K, on both sides of what was measured; only products that take them are noted as ones with bounded waits."""
    o = ops()
    for n, k in [(4096, 1024), (6144, 1024), (1024, 2048), (1024, 3072), (4096, 4096), (4096, 12288), (16384, 1024), (512, 1024)]:
        assert o._f32_takes_tc(n, k), (n, k)
    for n, k in [(512, 512), (3072, 512), (8192, 768), (1024, 1023), (2048, 2048), (19456, 2560), (32769, 1024), (151936, 1024)]:
        assert not o._f32_takes_tc(n, k), (n, k)
    o.check_device_errors()
    o.gemm_nt_simt(rnd((3, 512), torch.float32, 1), rnd((64, 512), torch.float32, 2))
    assert not o.bounded_wait_pending()
    o.gemm_nt_simt(rnd((3, 1024), torch.float32, 1), rnd((64, 1024), torch.float32, 2))
    assert o.bounded_wait_pending()
    o.check_device_errors()


@pytest.mark.parametrize("K", [512, 1024, 1100, 3072])
@pytest.mark.parametrize("M", [1, 37, 130])
def test_gemm_float32_tiny_operands_against_large_ones(M, K):
    """Operands below what bfloat16 parts hold against ones so large that their sums are ordinary numbers (or would be: all parts of the
    smallest are 0), beside ordinary rows: every sum within K roundings of 2^-24 of the sum of the products' magnitudes.  A row of zeros gives
    zeros; the ordinary rows have the bits that they have without the others."""
    a, w = rnd((M, K), torch.float32, 1), rnd((200, K), torch.float32, 2)
    plain = ops().gemm_nt_simt(a, w)
    w2 = w.clone()
    for n, size in enumerate([1e20, 1e25, 1e30, 1e12, 2.0 ** 29, 1e-20]):
        w2[3 + 20 * n] = (0.5 + rnd((K,), torch.float32, 5 + n).abs()) * size
    w2[7] = 0
    x = a.clone()
    small = [3e-38, 1e-40, 1e-42, 1e-36, 1e-33, 1e-25]
    for i, size in enumerate(small[:M]):
        x[i * (M // len(small))] = (0.5 + rnd((K,), torch.float32, 20 + i).abs()) * size
    got = ops().gemm_nt_simt(x, w2)
    X, W = f64(x), f64(w2)
    want, size = X @ W.T, abs(X) @ abs(W).T
    assert (size < 3e38).all()
    assert (abs(f64(got) - want) <= K * 2.0 ** -24 * size + K * 2.0 ** -149).all()
    assert (got[:, 7] == 0).all()
    rows = [m for m in range(M) if torch.equal(x[m], a[m])]
    cols = [n for n in range(200) if torch.equal(w2[n], w[n])]
    assert torch.equal(got[rows][:, cols], plain[rows][:, cols])


@pytest.mark.parametrize("M,N,K", [(1, 4096, 1024), (12, 1000, 777), (12, 1000, 1100), (40, 6144, 1024), (99, 4096, 1024), (3, 40000, 300)])
def test_gemm_float32_waits_for_a_w_that_was_just_written(M, N, K):
    """W written by the kernel launched just before, in memory that holds NaN until then: the products (plain, per head, of a batch)
    see it whole, as they do when the GPU was waited for in between; with `w_ready` and a W that is, the same bits."""
    a = rnd((M, K), torch.float32, 1)
    for seed in range(4):
        x = rnd((N, 2 * K), torch.float32, 10 + seed)
        w = ops().gated_act(x, "silu")
        torch.cuda.synchronize()
        want = ops().gemm_nt_simt(a, w, w_ready=True)

        def just_written():
            torch.full((N, K), float("nan"), device=DEV)   # (given back at once: the block that the next result of this size takes)
            return ops().gated_act(x, "silu")

        assert torch.equal(ops().gemm_nt_simt(a, just_written()), want)
        out = torch.empty((M, 1, N), device=DEV)
        ops().gemm_heads(a.view(M, 1, K), just_written().view(1, N, K), out)
        assert torch.equal(out[:, 0], want)
        assert torch.equal(ops().gemm_members(a.view(1, M, K), just_written().view(1, N, K))[0], want)


@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M,N,K,wide", [(1, 512, 128, 192), (8, 130, 512, 512), (5, 7, 32, 40), (3, 16, 96, 96), (8, 512, 192, 200), (2, 64, 256, 257), (7, 24, 384, 384),
                                        (8, 40, 160, 160), (4, 48, 520, 520)])
def test_gemm_heads_of_few_rows(M, N, K, wide, out_dtype):
    """Products per head of up to eight rows: every cut of k that the tensor cores take (whole, two and four parts), sizes and strides that they
    do not; heads inside wider rows of A and of the result.  float32 results: the error of float32 sums of k terms."""
    H = 3
    a, w = rnd((M, H, wide), torch.bfloat16, 1), rnd((H, N, K), torch.bfloat16, 2, 0.05)
    out = torch.full((M, H, N + 3), 7.0, dtype=out_dtype, device=DEV)
    ops().gemm_heads(a[:, :, :K], w, out[:, :, :N])
    want = np.einsum("mhk,hnk->mhn", f64(a[:, :, :K]), f64(w))
    if out_dtype == torch.float32:
        assert (abs(f64(out[:, :, :N]) - want) <= 2 * K * 2.0 ** -24 * np.einsum("mhk,hnk->mhn", abs(f64(a[:, :, :K])), abs(f64(w)))).all()
    else:
        close(out[:, :, :N], want, torch.bfloat16)
    assert (out[:, :, N:] == 7.0).all()


TURNED_SHAPES = [(1, 16, 1, 0, 1), (2, 32, 1, 0, 2), (1, 48, 5, 0, 2), (2, 64, 4, 0, 1), (1, 112, 8, 0, 1), (1, 128, 1, 0, 2), (2, 160, 1, 32, 1),
                 (2, 256, 3, 0, 1), (1, 240, 1, 16, 1), (2, 208, 1, 64, 1)]     # blocks of a tile, rows of A, runs of k, rows of the last W tiles, blocks an SM


@pytest.mark.parametrize("M,N,K", [(9, 256, 64), (16, 2064, 1032), (33, 400, 520), (64, 1040, 1000), (65, 16, 8), (312, 2576, 1088), (777, 528, 256), (800, 19456, 72)])
def test_gemm_turned(M, N, K):
    """The turned product with every kind of tile, and with the one that is chosen: rows and columns that no tile divides, k that no block of 64
    divides, fewer W tiles than the rest with narrow ones; plain and gated, both results.  Rows of NaN behind a and w are not read."""
    a = torch.full((M + 8, K), float("nan"), dtype=torch.bfloat16, device=DEV)
    w = torch.full((N + 16, K), float("nan"), dtype=torch.bfloat16, device=DEV)
    a[:M], w[:N] = rnd((M, K), torch.bfloat16, 6), rnd((N, K), torch.bfloat16, 7, 0.05)
    a, w = a[:M], w[:N]
    want = f64(a) @ f64(w).T
    g = want.reshape(M, N // 16, 2, 8)
    gated = (P.silu(g[:, :, 0]) * g[:, :, 1]).reshape(M, N // 2)
    error, lib, stream = torch.zeros(1, dtype=torch.int32, device=DEV), ops().library(), ops()._stream()
    for cg, n, runs, narrow, per_sm in TURNED_SHAPES:
        runs = min(runs, -(-K // 64))
        full = max(0, -(-N // (128 * cg)) - 2)
        for is_gated, dtype in ((0, torch.bfloat16), (1, torch.bfloat16), (0, torch.float32), (1, torch.float32)):
            out = torch.full((M, N // 2 if is_gated else N), float("nan"), dtype=dtype, device=DEV)
            assert lib.vx_gemm_turned_shape(a.data_ptr(), w.data_ptr(), out.data_ptr(), M, N, K, K, K, out.shape[1], is_gated, 0, ops().dtype_code(dtype), 1,
                                            cg, n, runs, full, narrow, per_sm, error.data_ptr(), stream) == 0
            close(out, gated if is_gated else want, torch.bfloat16, what=str((cg, n, runs, narrow, per_sm)))
    for dtype in (torch.bfloat16, torch.float32):
        close(ops().gemm_turned(a, w, dtype), want, torch.bfloat16)
        close(ops().gemm_turned(a, w, dtype, gated_activation="silu", w_ready=True), gated, torch.bfloat16)
    assert int(error.item()) == 0
    ops().check_device_errors()


@pytest.mark.parametrize("M,N,K", [(24, 24576, 512), (24, 2560, 4096), (50, 12288, 512), (150, 6144, 1024), (312, 4096, 2048)])
def test_gemm_turned_waits_for_a_w_that_was_just_written(M, N, K):
    """W written by the kernel launched just before, in memory that holds NaN until then: without `w_ready` the product sees it whole, with every
    kind of tile that is chosen; with `w_ready` and a W that is, the same bits."""
    a = rnd((M, K), torch.bfloat16, 1)
    for seed in range(4):
        x = rnd((N, 2 * K), torch.float32, 10 + seed)
        w = ops().gated_act(x, "silu", out_dtype=torch.bfloat16)
        torch.cuda.synchronize()
        want = [ops().gemm_turned(a, w, w_ready=True), ops().gemm_turned(a, w, gated_activation="silu", w_ready=True)]

        def just_written():
            torch.full((N, K), float("nan"), dtype=torch.bfloat16, device=DEV)   # (given back at once: the block that the next result of this size takes)
            return ops().gated_act(x, "silu", out_dtype=torch.bfloat16)

        assert torch.equal(ops().gemm_turned(a, just_written()), want[0])
        assert torch.equal(ops().gemm_turned(a, just_written(), gated_activation="silu"), want[1])
    ops().check_device_errors()


@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M,N,K", [(1, 53, 72), (37, 64, 16), (130, 136, 104), (64, 384, 96), (8, 4096, 4096)])
def test_gemm_bf16(M, N, K, out_dtype):
    a, w = rnd((M, K), torch.bfloat16, 6), rnd((N, K), torch.bfloat16, 7, 0.05)
    want = f64(a) @ f64(w).T
    close(ops().gemm_bf16(a, w, None, out_dtype), want, torch.bfloat16)
    close(ops().gemm_nt_simt(a, w, None, out_dtype), want, torch.bfloat16)  # the plain product takes bfloat16 too
    bias = rnd((N,), torch.float32, 8)
    close(ops().gemm_bf16(a, w, bias, out_dtype), want + f64(bias), torch.bfloat16)


# ----------------------------------------------------------------------------
def test_sample_greedy_ties_and_rows():
    x = torch.randn(5, 1000, generator=torch.Generator().manual_seed(0)).to(DEV)
    x[2, 77] = x[2, 400] = 9.0  # the first maximum wins
    got = ops().sample(x).tolist()
    assert got == [P.greedy(r) for r in f64(x)] and got[2] == 77
    wide = torch.randn(3, 151936, generator=torch.Generator().manual_seed(1)).to(DEV)
    assert ops().sample(wide).tolist() == wide.argmax(-1).tolist()


@pytest.mark.parametrize("vocab", [384, 5000, 151936])
def test_sample_temperature_and_top_p(vocab):
    from velox_b200.sampling.rng import uniform
    rows = 12
    x = (torch.randn(rows, vocab, generator=torch.Generator().manual_seed(2)) * 2.0).to(DEV)
    temps = [0.0, 0.8, 1.0, 0.5, 1.3, 0.8, 0.8, 1.0, 0.0, 0.7, 2.0, 0.8]
    tops = [1.0, 1.0, 0.9, 0.5, 1.0, 0.3, 0.95, 0.0, 0.5, 0.999, 0.8, 1.0]
    us = [uniform(5, 0, i) for i in range(rows)]
    t = lambda v: torch.tensor(v, dtype=torch.float32, device=DEV)
    got = ops().sample(x, t(temps), t(tops), t(us)).tolist()
    xs = f64(x)
    for r in range(rows):
        if temps[r] <= 1e-7:
            assert got[r] == P.greedy(xs[r])
            continue
        p = P.probabilities(xs[r], temps[r], tops[r])
        want = P.sample_from(p, us[r])
        if got[r] != want:
            # float32 against float64 may disagree only where u falls on a boundary of the
            # cumulative distribution, or where the nucleus' edge is a near-tie
            c = np.cumsum(p)
            lo, hi = sorted((got[r], want))
            assert p[got[r]] > 0 and abs(c[lo] - us[r]) < 1e-5 * max(1, hi - lo), (r, got[r], want)
    # the same inputs give the same tokens
    assert ops().sample(x, t(temps), t(tops), t(us)).tolist() == got


@pytest.mark.parametrize("vocab", [25000, 60001, 151936, 262144])
def test_sample_gives_the_same_token_in_every_form(vocab):
    """On a B200 1 and 12 rows are drawn by eight blocks a row, 20 by four, 40 by two and 80 by one (fewer where the vocabulary is
    small), with the row's parts kept in shared memory or, where they don't fit or nothing is drawn, read again.  Every form adds in the same order, so a
    row's token is the same in all of them, bit for bit, and each form is held against float64.  60,001: rows that begin on no 16-byte
    address.  Ties of the maximum lie in different blocks' parts."""
    from velox_b200.sampling.rng import uniform
    rows = 80
    x = torch.randn(rows, vocab, generator=torch.Generator().manual_seed(vocab)) * 2.0
    for r in range(0, rows, 4):
        x[r, [vocab // 3 + r, vocab - 1 - r]] = 20.0   # (the first wins)
    temps = [(0.0, 0.8, 1.0, 1.3)[r % 4] for r in range(rows)]
    tops = [(1.0, 0.9, 0.5, 0.0, 0.999)[r % 5] for r in range(rows)]
    us = [uniform(7, 0, r) for r in range(rows)]
    x, t = x.to(DEV), lambda v: torch.tensor(v, dtype=torch.float32, device=DEV)
    draw = lambda n: ops().sample(x[:n], t(temps[:n]), t(tops[:n]), t(us[:n])).tolist()
    got = draw(rows)
    for n in (1, 12, 20, 40):
        assert draw(n) == got[:n], n
        assert ops().sample(x[:n]).tolist() == [P.greedy(v) for v in f64(x[:n])], n
    assert ops().sample(x).tolist() == [P.greedy(v) for v in f64(x)]
    assert all(got[r] == vocab // 3 + r for r in range(0, rows, 4))
    for r in range(1, 40):
        if temps[r] == 0.0:
            continue
        p = P.probabilities(f64(x[r]), temps[r], tops[r])
        want = P.sample_from(p, us[r])
        if got[r] != want:   # only where u falls on a boundary of the cumulative distribution (as above)
            c = np.cumsum(p)
            lo, hi = sorted((got[r], want))
            assert p[got[r]] > 0 and abs(c[lo] - us[r]) < 1e-5 * max(1, hi - lo), (r, got[r], want)


def test_sample_top_p_keeps_only_the_nucleus():
    x = torch.full((1, 300), -5.0, device=DEV)
    x[0, [10, 20, 30]] = torch.tensor([3.0, 2.0, 1.0], device=DEV)
    t = lambda v: torch.tensor([v], dtype=torch.float32, device=DEV)
    seen = set()
    for i in range(64):
        seen.add(ops().sample(x, t(1.0), t(0.85), t(i / 64.0)).item())
    assert seen == {10, 20}  # p = .66, .24, .09: the first two reach 0.85
    assert {ops().sample(x, t(1.0), t(0.5), t(i / 64.0)).item() for i in range(64)} == {10}
    # ties at the nucleus' edge stay together: p = .475, .175 x 3, the rest 0.002 in all; 0.6 is crossed inside the tie
    y = torch.full((1, 5000), -12.0, device=DEV)
    y[0, [7, 4000, 4500, 4999]] = torch.tensor([3.0, 2.0, 2.0, 2.0], device=DEV)
    seen = {ops().sample(y, t(1.0), t(0.6), t(i / 256.0)).item() for i in range(256)}
    assert seen == {7, 4000, 4500, 4999}
    p = P.probabilities(f64(y)[0], 1.0, 0.6)
    assert set(np.nonzero(p)[0].tolist()) == seen


# ----------------------------------------------------------------------------
DECODE_CASES = [
    # (kv lengths, H, Hk, D, S, window)
    ([1, 2, 15, 16, 17], 8, 2, 128, 16, 0),          # first tokens, around a page's edge
    ([255, 256, 257, 600, 1600], 8, 2, 128, 16, 0),   # around a piece's edge (256 keys), several pieces
    ([700, 33, 300], 6, 6, 64, 32, 0),               # no grouping, head size 64, pages of 32
    ([900, 64, 257], 16, 1, 64, 16, 0),              # 16 query heads share one kv head
    ([1300, 40, 590, 5], 4, 2, 128, 16, 540),        # a window that crosses split boundaries
    ([3000], 32, 8, 128, 16, 0),                     # the flagship's head layout, 12 pieces
    # more pieces than SMs: a warp per piece (above, a block of eight warps per piece)
    ([1000] + [(i * 97) % 1000 + 1 for i in range(19)], 16, 8, 128, 16, 0),   # 640 pieces
    ([1000] + [(i * 61) % 1000 + 1 for i in range(25)], 16, 8, 128, 16, 0),   # 832 pieces
    ([1000] + [(i * 43) % 1000 + 1 for i in range(29)], 16, 8, 64, 16, 0),    # 960 pieces, heads of 64
    # two pieces at most: the first ones before the second ones
    ([512, 257, 256, 1] + [(i * 37) % 512 + 1 for i in range(20)], 16, 8, 128, 16, 0),
    ([900, 300, 256, 7] + [(i * 91) % 900 + 1 for i in range(30)], 16, 4, 64, 32, 300),   # (a window of 300 keys)
]


@pytest.mark.parametrize("case", range(len(DECODE_CASES)))
def test_paged_decode_attention(case):
    lens, H, Hk, D, S, window = DECODE_CASES[case]
    seqs = [(n - 1, 1) for n in lens]
    q, kp, vp, bt, sot, pos, want = paged_case(torch.bfloat16, seqs, H, Hk, D, S, window, seed=40 + case)
    out = ops().paged_decode_attention(q, H * D, kp, vp, bt, sot, pos, 1 / math.sqrt(D), window, H, Hk, D,
                                       len(lens), max(lens))
    close(out, want, torch.bfloat16, what="decode attention case %d" % case)
    # and it agrees with the general kernel far more closely than with the bound
    gen = ops().paged_attention_generic(q, H * D, kp, vp, bt, sot, pos, 1 / math.sqrt(D), window, H, Hk, D, len(lens))
    assert (out.float() - gen.float()).abs().max() < 2e-2


@pytest.mark.parametrize("far", [0, 17, 255, 256, 700, 1023])
def test_decode_attention_finds_one_far_key(far):
    H, Hk, D, S = 8, 2, 128, 16
    q, kp, vp, bt, sot, pos, want = paged_case(torch.bfloat16, [(1099, 1)], H, Hk, D, S, 0, seed=12, spike=far)
    out = ops().paged_decode_attention(q, H * D, kp, vp, bt, sot, pos, 1 / math.sqrt(D), 0, H, Hk, D, 1, 1100)
    close(out, want, torch.bfloat16)
    page, off = int(bt[0, far // S]), far % S
    assert torch.allclose(out[0, :D].float(), vp[page, 0, off].float(), atol=5e-2)


def test_decode_attention_token_rows_and_batch_independence():
    """Requests picked out of a larger batch by row; a request's output does not
    depend on which others are beside it."""
    H, Hk, D, S = 8, 2, 128, 16
    seqs = [(0, 5), (499, 1), (0, 3), (299, 1), (1200, 1)]
    q, kp, vp, bt, sot, pos, want = paged_case(torch.bfloat16, seqs, H, Hk, D, S, 0, seed=13)
    rows = torch.tensor([5, 9, 10], dtype=torch.int32, device=DEV)  # the three single-token requests
    out = torch.zeros((11, H * D), dtype=torch.bfloat16, device=DEV)
    ops().paged_decode_attention(q, H * D, kp, vp, bt, sot, pos, 1 / math.sqrt(D), 0, H, Hk, D, 3, 1201,
                                 token_rows=rows, out=out)
    close(out[rows.long()], want[[5, 9, 10]], torch.bfloat16)
    assert (out[:5] == 0).all()
    alone = torch.zeros_like(out)
    ops().paged_decode_attention(q, H * D, kp, vp, bt, sot, pos, 1 / math.sqrt(D), 0, H, Hk, D, 1, 500,
                                 token_rows=rows[:1], out=alone)
    assert torch.equal(alone[5], out[5])  # bit-identical alone and in company


def test_decode_attention_gives_the_same_bits_in_every_block_shape():
    """The kernel gives a piece a block of eight warps or one warp, by the step's size; a request's
    output must not notice (1 request has fewer pieces than a GPU has SMs, 20, 26 and 30 have more)."""
    H, Hk, D, S = 16, 8, 128, 16
    lens = [1000] + [(i * 43) % 1000 + 1 for i in range(29)]
    q, kp, vp, bt, sot, pos, want = paged_case(torch.bfloat16, [(n - 1, 1) for n in lens], H, Hk, D, S, 0, seed=15)
    full = ops().paged_decode_attention(q, H * D, kp, vp, bt, sot, pos, 1 / math.sqrt(D), 0, H, Hk, D, 30, 1000)
    close(full, want, torch.bfloat16)
    for n in (1, 20, 26):
        part = ops().paged_decode_attention(q, H * D, kp, vp, bt, sot, pos, 1 / math.sqrt(D), 0, H, Hk, D, n, 1000)
        assert torch.equal(part[:n], full[:n]), n


@pytest.mark.parametrize("D,H,Hk,window,S", [(128, 8, 2, 0, 16), (128, 24, 2, 0, 32), (64, 6, 6, 300, 16), (64, 32, 2, 0, 48)])
def test_decode_attention_forms_agree(D, H, Hk, window, S):
    """A block or a warp per piece: the same bits, at lengths around the edges of a tile (16 keys), a sub-piece (32), the
    ring (64) and a piece (256), with one and two tiles of 8 query heads."""
    lens = [1, 16, 17, 32, 33, 64, 65, 96, 97, 224, 255, 256, 257, 289, 513, 800]
    q, kp, vp, bt, sot, pos, want = paged_case(torch.bfloat16, [(n - 1, 1) for n in lens], H, Hk, D, S, window, seed=17)
    run = lambda shape: ops().paged_decode_attention(q, H * D, kp, vp, bt, sot, pos, 1 / math.sqrt(D), window, H, Hk, D, len(lens),
                                                     max(lens), shape=shape)
    first = run(0)
    close(first, want, torch.bfloat16)
    for shape in (1, 8):
        assert torch.equal(run(shape), first), shape


@pytest.mark.parametrize("D,H,Hk,window", [(128, 8, 2, 0), (64, 16, 1, 0), (128, 6, 6, 333)])
def test_decode_attention_in_pieces_of_any_number_of_tiles(D, H, Hk, window):
    """The C entry points take 1 to 32 tiles of 16 keys a piece: even numbers, odd ones (whose last sub-piece is half of one, with
    another piece's keys behind it) and more tiles than a request has."""
    S, lens = 16, [600, 16, 33, 257, 40, 5]
    q, kp, vp, bt, sot, pos, want = paged_case(torch.bfloat16, [(n - 1, 1) for n in lens], H, Hk, D, S, window, seed=19)
    stream, no_alloc = torch.cuda.current_stream().cuda_stream, ops().library().vx_paged_decode_attention_static
    ptr, num, real = ctypes.c_void_p, ctypes.c_int, ctypes.c_float
    no_alloc.argtypes = [ptr, num, ptr, ptr, ptr, num, ptr, ptr, ptr, num, ptr, num, real] + [num] * 7 + [ptr]
    for tiles in (1, 2, 3, 5, 15, 16, 31, 32):
        pieces = -(-(-(-max(lens) // 16)) // tiles) + (1 if window else 0)
        scratch = torch.full((len(lens) * H * pieces * (D + 2),), float("nan"), device=DEV)
        args = (q.data_ptr(), H * D, kp.data_ptr(), vp.data_ptr(), bt.data_ptr(), bt.shape[1], None, sot.data_ptr(), pos.data_ptr())
        rest = (H * D, 1 / math.sqrt(D), window, len(lens), H, Hk, D, S, tiles)
        out, static = torch.zeros((len(lens), H * D), dtype=torch.bfloat16, device=DEV), torch.zeros((len(lens), H * D), dtype=torch.bfloat16, device=DEV)
        assert ops().library().vx_paged_decode_attention(*args, scratch.data_ptr(), pieces, out.data_ptr(), *rest, 1, stream) == 0
        close(out, want, torch.bfloat16, what="%d tiles a piece" % tiles)
        assert no_alloc(*args, pieces, static.data_ptr(), *rest, stream) == 0
        assert torch.equal(static, out), tiles


def test_decode_attention_shows_a_score_that_is_no_number():
    """A query that is not a number gives an output that is none, whatever the number of keys; its neighbours keep theirs."""
    H, Hk, D, S = 8, 2, 128, 16
    lens = [1, 33, 257, 700]
    q, kp, vp, bt, sot, pos, _ = paged_case(torch.bfloat16, [(n - 1, 1) for n in lens], H, Hk, D, S, 0, seed=18)
    good = ops().paged_decode_attention(q, H * D, kp, vp, bt, sot, pos, 0.1, 0, H, Hk, D, 4, 700)
    q2 = q.clone()
    q2.view(4, H, D)[:, 3, 5] = float("nan")
    got = ops().paged_decode_attention(q2, H * D, kp, vp, bt, sot, pos, 0.1, 0, H, Hk, D, 4, 700).view(4, H, D)
    assert torch.isnan(got[:, 3]).all()
    rest = [h for h in range(H) if h != 3]
    assert torch.equal(got[:, rest], good.view(4, H, D)[:, rest])


def test_decode_attention_refuses_what_it_cannot_do():
    from velox_b200.csrc.ops import KernelError
    q, kp, vp, bt, sot, pos, _ = paged_case(torch.bfloat16, [(9, 1)], 4, 2, 48, 16, 0, seed=14)
    with pytest.raises(KernelError, match="size"):
        ops().paged_decode_attention(q, 4 * 48, kp, vp, bt, sot, pos, 0.1, 0, 4, 2, 48, 1, 10)
    assert not ops().decode_attention_supported(torch.bfloat16, 48, 16, 2)
    assert not ops().decode_attention_supported(torch.bfloat16, 128, 8, 2)
    assert not ops().decode_attention_supported(torch.float32, 128, 16, 2)


# ----------------------------------------------------------------------------
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M,N,K", [(1, 48, 64), (3, 50, 96), (8, 4096, 4096), (7, 136, 160), (8, 333, 1024), (5, 16, 12288)])
def test_gemm_skinny(M, N, K, out_dtype):
    a, w = rnd((M, K), torch.bfloat16, 20), rnd((N, K), torch.bfloat16, 21, 0.05)
    bias = rnd((N,), torch.float32, 22)
    want = f64(a) @ f64(w).T
    close(ops().gemm_skinny(a, w, None, out_dtype), want, torch.bfloat16, what="skinny")
    close(ops().gemm_skinny(a, w, bias, out_dtype), want + f64(bias), torch.bfloat16, what="skinny + bias")
    # against the plain product on the same bfloat16 inputs: only the order of additions differs
    ref = ops().gemm_nt_simt(a, w, None, torch.float32)
    got = ops().gemm_skinny(a, w, None, torch.float32)
    assert (got - ref).abs().max() <= 1e-3 * max(1.0, float(ref.abs().max()))
    # a row alone gives the same bits as in company
    alone = ops().gemm_skinny(a[:1].contiguous(), w, None, torch.float32)
    assert torch.equal(alone[0], got[0])


@pytest.mark.parametrize("act", ["silu", "gelu_pytorch_tanh"])
@pytest.mark.parametrize("M,I,K", [(2, 24, 64), (8, 200, 96), (5, 1024, 512)])
def test_gemm_skinny_gated(M, I, K, act):
    a = rnd((M, K), torch.bfloat16, 23)
    wg, wu = rnd((I, K), torch.bfloat16, 24, 0.1), rnd((I, K), torch.bfloat16, 25, 0.1)
    # tiles of 16 rows: 8 gate rows, then their 8 up rows
    w = torch.stack([wg.view(I // 8, 8, K), wu.view(I // 8, 8, K)], 1).reshape(2 * I, K).contiguous()
    g, u = f64(a) @ f64(wg).T, f64(a) @ f64(wu).T
    av = P.silu(g) if act == "silu" else 0.5 * g * (1 + np.tanh(math.sqrt(2 / math.pi) * (g + 0.044715 * g ** 3)))
    close(ops().gemm_skinny(a, w, None, torch.bfloat16, gated_activation=act), av * u, torch.bfloat16, what="gated")


def test_gemm_skinny_refuses_what_it_cannot_do():
    from velox_b200.csrc.ops import KernelError
    a, w = rnd((9, 64), torch.bfloat16, 1), rnd((32, 64), torch.bfloat16, 2)
    with pytest.raises(KernelError):
        ops().gemm_skinny(a, w)
    with pytest.raises(KernelError):
        ops().gemm_skinny(rnd((4, 40), torch.bfloat16, 1), rnd((32, 40), torch.bfloat16, 2))
    assert not ops().skinny_supported(4, 40, a, w) and not ops().skinny_supported(9, 64, a, w)


# ----------------------------------------------------------------------------
def prefill_inputs(seqs):
    cu = np.concatenate([[0], np.cumsum([n for _, n in seqs])]).astype(np.int32)
    offs = np.asarray([o for o, _ in seqs], np.int32)
    return torch.from_numpy(cu).to(DEV), torch.from_numpy(offs).to(DEV)


PREFILL_CASES = [
    # (seqs (kv_offset, new tokens), H, Hk, D, S, window)
    ([(0, 1)], 4, 2, 64, 16, 0),                               # a sequence's first token
    ([(0, 64)], 4, 2, 128, 16, 0),                             # exactly one tile
    ([(0, 65), (0, 3), (0, 127)], 4, 4, 128, 16, 0),           # one past a tile, a short one, one short of two tiles
    ([(0, 8), (20, 4), (10, 1)], 8, 2, 64, 16, 0),             # the reference's mixed batch: cold 8, warm 4 @20, decode 1 @10
    ([(100, 200), (63, 2), (64, 1), (300, 1)], 8, 2, 128, 16, 0),   # portions on top of cached keys, decodes beside them
    ([(0, 300)], 6, 3, 64, 32, 0),                             # pages of 32, 3 groups
    ([(0, 200), (150, 90), (400, 1)], 4, 1, 128, 16, 70),      # a window that is no multiple of the tile
    ([(7, 130)], 32, 8, 128, 16, 0),                           # the flagship's head layout
]


@pytest.mark.parametrize("case", range(len(PREFILL_CASES)))
def test_paged_prefill_attention(case):
    seqs, H, Hk, D, S, window = PREFILL_CASES[case]
    q, kp, vp, bt, sot, pos, want = paged_case(torch.bfloat16, seqs, H, Hk, D, S, window, seed=60 + case)
    cu, offs = prefill_inputs(seqs)
    out = ops().paged_prefill_attention(q, H * D, kp, vp, bt, cu, offs, 1 / math.sqrt(D), window, H, Hk, D,
                                        len(seqs), max(n for _, n in seqs), q.shape[0])
    close(out, want, torch.bfloat16, what="prefill attention case %d" % case)
    gen = ops().paged_attention_generic(q, H * D, kp, vp, bt, sot, pos, 1 / math.sqrt(D), window, H, Hk, D, q.shape[0])
    assert (out.float() - gen.float()).abs().max() < 2e-2


@pytest.mark.parametrize("far", [0, 63, 64, 500, 777])
def test_prefill_attention_finds_one_far_key(far):
    H, Hk, D, S = 8, 2, 128, 16
    seqs = [(700, 100)]
    q, kp, vp, bt, sot, pos, want = paged_case(torch.bfloat16, seqs, H, Hk, D, S, 0, seed=15, spike=far)
    cu, offs = prefill_inputs(seqs)
    out = ops().paged_prefill_attention(q, H * D, kp, vp, bt, cu, offs, 1 / math.sqrt(D), 0, H, Hk, D, 1, 100, 100)
    close(out, want, torch.bfloat16)
    page, off = int(bt[0, far // S]), far % S
    assert torch.allclose(out[-1, :D].float(), vp[page, 0, off].float(), atol=5e-2)  # the last query has the spike


# ----------------------------------------------------------------------------
TC_SHAPES = [(128, 256, 64), (128, 128, 128), (256, 512, 4096), (200, 384, 96), (77, 48, 72), (1000, 6144, 4096),
             (2048, 4096, 12288)]


TC_TILES = {"128x256": dict(wide=True), "128x128": dict(wide=False), "256x256 by a pair of blocks": dict(pair=True)}


@pytest.mark.parametrize("tiles", list(TC_TILES))
@pytest.mark.parametrize("M,N,K", TC_SHAPES)
def test_gemm_tcgen05(M, N, K, tiles):
    how = TC_TILES[tiles]
    a, w = rnd((M, K), torch.bfloat16, 30), rnd((N, K), torch.bfloat16, 31, 0.05)
    got = ops().gemm_tcgen05(a, w, None, **how)
    ops().check_device_errors()
    if M * N * K <= 1 << 28:
        close(got, f64(a) @ f64(w).T, torch.bfloat16, what="tcgen05")
    # against the library product on the same inputs (both accumulate in float32)
    ref = torch.mm(a, w.t())
    scale = max(1.0, float(ref.float().abs().max()))
    assert (got.float() - ref.float()).abs().max() <= 2e-2 * scale
    bias = rnd((N,), torch.float32, 32)
    got_b = ops().gemm_tcgen05(a, w, bias, **how)
    assert (got_b.float() - (ref.float() + bias)).abs().max() <= 2e-2 * scale + 2e-2


@pytest.mark.parametrize("tiles", list(TC_TILES))
@pytest.mark.parametrize("M,I,K", [(128, 128, 64), (300, 200, 96), (2048, 12288, 4096)])
def test_gemm_tcgen05_gated(M, I, K, tiles):
    a = rnd((M, K), torch.bfloat16, 33)
    wg, wu = rnd((I, K), torch.bfloat16, 34, 0.05), rnd((I, K), torch.bfloat16, 35, 0.05)
    w = torch.stack([wg.view(I // 8, 8, K), wu.view(I // 8, 8, K)], 1).reshape(2 * I, K).contiguous()
    got = ops().gemm_tcgen05(a, w, None, gated_activation="silu", **TC_TILES[tiles])
    ops().check_device_errors()
    g, u = torch.mm(a, wg.t()).float(), torch.mm(a, wu.t()).float()
    want = torch.nn.functional.silu(g) * u
    assert got.shape == (M, I)
    assert (got.float() - want).abs().max() <= 3e-2 + 3e-2 * float(want.abs().max())


# ----------------------------------------------------------------------------
TC_PREFILL_CASES = [
    ([(0, 1)], 4, 2, 128, 16, 0),                                  # a sequence's first token
    ([(0, 128)], 4, 1, 128, 16, 0),                                # 4 heads share a tile: 32 tokens each
    ([(0, 65), (0, 3), (0, 127)], 4, 4, 128, 16, 0),               # no sharing: 128 tokens a tile
    ([(100, 200), (63, 2), (64, 1), (300, 1)], 8, 2, 128, 16, 0),  # portions on top of cached keys, decodes beside them
    ([(0, 300)], 16, 2, 128, 32, 0),                               # 8 heads share, pages of 32
    ([(0, 400), (350, 90), (600, 1)], 4, 1, 128, 16, 170),         # a window that is no multiple of the tile
    ([(0, 300), (77, 41)], 10, 2, 128, 16, 0),                     # 5 heads a kv head (24 tokens of each in a tile, 8 rows idle)
    ([(130, 100), (0, 50)], 3, 1, 128, 32, 90),                    # 3 heads: 40 tokens each; a window
    ([(0, 200)], 14, 2, 128, 16, 0),                               # 7 heads: 16 tokens each, 16 rows idle
    ([(500, 64)], 6, 1, 128, 16, 0),                               # 6 heads
    ([(7, 333)], 32, 8, 128, 16, 0),                               # the flagship's head layout
    ([(0, 700)], 2, 1, 128, 16, 0),                                # two heads share: several tiles deep
]


@pytest.mark.parametrize("case", range(len(TC_PREFILL_CASES)))
def test_paged_prefill_attention_tc(case):
    seqs, H, Hk, D, S, window = TC_PREFILL_CASES[case]
    q, kp, vp, bt, sot, pos, want = paged_case(torch.bfloat16, seqs, H, Hk, D, S, window, seed=80 + case)
    cu, offs = prefill_inputs(seqs)
    out = ops().paged_prefill_attention_tc(q, H * D, kp, vp, bt, cu, offs, 1 / math.sqrt(D), window, H, Hk, D,
                                           len(seqs), max(n for _, n in seqs), q.shape[0])
    ops().check_device_errors()
    close(out, want, torch.bfloat16, what="tcgen05 prefill attention case %d" % case)
    gen = ops().paged_attention_generic(q, H * D, kp, vp, bt, sot, pos, 1 / math.sqrt(D), window, H, Hk, D, q.shape[0])
    assert (out.float() - gen.float()).abs().max() < 3e-2


@pytest.mark.parametrize("far", [0, 127, 128, 500, 777])
def test_prefill_attention_tc_finds_one_far_key(far):
    H, Hk, D, S = 8, 2, 128, 16
    seqs = [(700, 100)]
    q, kp, vp, bt, sot, pos, want = paged_case(torch.bfloat16, seqs, H, Hk, D, S, 0, seed=16, spike=far)
    cu, offs = prefill_inputs(seqs)
    out = ops().paged_prefill_attention_tc(q, H * D, kp, vp, bt, cu, offs, 1 / math.sqrt(D), 0, H, Hk, D, 1, 100, 100)
    ops().check_device_errors()
    close(out, want, torch.bfloat16)
    page, off = int(bt[0, far // S]), far % S
    assert torch.allclose(out[-1, :D].float(), vp[page, 0, off].float(), atol=5e-2)


# ----------------------------------------------------------------------------
def _attend(kernel, q, kp, vp, bt, sot, pos, seqs, H, Hk, D, window):
    scale = 1 / math.sqrt(D)
    if kernel == "generic":
        return ops().paged_attention_generic(q, H * D, kp, vp, bt, sot, pos, scale, window, H, Hk, D, q.shape[0])
    if kernel == "decode":
        return ops().paged_decode_attention(q, H * D, kp, vp, bt, sot, pos, scale, window, H, Hk, D, len(seqs),
                                            max(o + n for o, n in seqs))
    cu, offs = prefill_inputs(seqs)
    fn = ops().paged_prefill_attention_tc if kernel == "prefill_tc" else ops().paged_prefill_attention
    out = fn(q, H * D, kp, vp, bt, cu, offs, scale, window, H, Hk, D, len(seqs), max(n for _, n in seqs), q.shape[0])
    ops().check_device_errors()
    return out


@pytest.mark.parametrize("window,length", [(70, 400), (256, 1000), (33, 34), (129, 700)])
@pytest.mark.parametrize("kernel", ["generic", "decode", "prefill", "prefill_tc"])
def test_a_window_ends_where_it_should(kernel, window, length):
    """The query at position p sees the keys p + 1 - W to p (src/paged/metal_kernels.rs:135-137,
    339-341).  A key whose score towers over all others decides the output when it stands at
    p + 1 - W, and must leave no trace when it stands at p - W, one place further back."""
    H, Hk, D, S = 8, 2, 128, 16
    new = 1 if kernel == "decode" else min(40, length)      # the last query of a portion, or a decoded token
    seqs = [(length - new, new)]
    p = length - 1
    for inside in (True, False):
        j = p + 1 - window if inside else p - window
        q, kp, vp, bt, sot, pos, want = paged_case(torch.bfloat16, seqs, H, Hk, D, S, window, seed=17, spike=j)
        out = _attend(kernel, q, kp, vp, bt, sot, pos, seqs, H, Hk, D, window)
        close(out, want, torch.bfloat16, what="%s, spike %s the window" % (kernel, "inside" if inside else "behind"))
        value = vp[int(bt[0, j // S]), 0, j % S].float()
        near = torch.allclose(out[-1, :D].float(), value, atol=2e-2)
        assert near == inside, "%s: the key at %d (query at %d, window %d) %s" % (
            kernel, j, p, window, "was not seen" if inside else "was seen")


# ----------------------------------------------------------------------------
TC_SPLIT_CASES = [
    ([(3000, 64)], 8, 2, 128, 16, 0),                              # two query tiles on 24 key tiles: cut into 6 runs
    ([(1500, 40), (20, 33), (2500, 35), (0, 70)], 8, 2, 128, 16, 0),  # cut (3 runs), whole, cut (5 runs), whole, in one launch
    ([(2000, 100)], 32, 8, 128, 16, 0),                            # the flagship's head layout: 4 query tiles x 8 kv heads
    ([(4000, 50), (900, 60)], 4, 1, 128, 32, 600),                 # a window: the runs' tiles start far from key 0
    ([(1021, 130)], 4, 4, 128, 16, 0),                             # no sharing; the last tokens see one key tile more than the first
    ([(2100, 70), (1300, 33)], 10, 2, 128, 16, 0),                 # 5 heads a kv head, cut
]


@pytest.mark.parametrize("case", range(len(TC_SPLIT_CASES)))
def test_paged_prefill_attention_tc_cut_into_runs(case):
    """A short portion on top of many cached keys: its key tiles are cut into runs that several blocks take,
    and a second kernel adds the runs."""
    seqs, H, Hk, D, S, window = TC_SPLIT_CASES[case]
    q, kp, vp, bt, sot, pos, want = paged_case(torch.bfloat16, seqs, H, Hk, D, S, window, seed=120 + case)
    cu, offs = prefill_inputs(seqs)
    max_kv = max(o + n for o, n in seqs)
    out = ops().paged_prefill_attention_tc(q, H * D, kp, vp, bt, cu, offs, 1 / math.sqrt(D), window, H, Hk, D,
                                           len(seqs), max(n for _, n in seqs), q.shape[0], max_kv=max_kv)
    ops().check_device_errors()
    close(out, want, torch.bfloat16, what="tcgen05 prefill attention in runs, case %d" % case)
    whole = ops().paged_prefill_attention_tc(q, H * D, kp, vp, bt, cu, offs, 1 / math.sqrt(D), window, H, Hk, D,
                                             len(seqs), max(n for _, n in seqs), q.shape[0])
    assert not torch.equal(out, whole), "nothing was cut: the case lost its point"
    assert (out.float() - whole.float()).abs().max() < 2e-2
    # a request's result does not depend on what else is in the launch
    if len(seqs) > 1:
        alone_q, kp1, vp1, bt1, _, _, _ = paged_case(torch.bfloat16, seqs[:1], H, Hk, D, S, window, seed=120 + case)
        cu1, offs1 = prefill_inputs(seqs[:1])
        alone = ops().paged_prefill_attention_tc(alone_q, H * D, kp1, vp1, bt1, cu1, offs1, 1 / math.sqrt(D), window, H, Hk,
                                                 D, 1, seqs[0][1], alone_q.shape[0], max_kv=max_kv)
        assert torch.equal(alone, out[:seqs[0][1]])


@pytest.mark.parametrize("seed", range(10))
def test_paged_prefill_attention_tc_drawn_shapes(seed):
    """Drawn cases: one to four requests with portions of 1 to 400 tokens on 0 to 3,000 cached keys, every group size (1 to 8)
    and page size the kernel takes, with and without a window (of any length, so that the two query tiles of a block
    want different key tiles), cut into runs or not.  Never-written slots of the pools hold NaN."""
    rng = np.random.default_rng(900 + seed)
    G = int(rng.choice([1, 2, 3, 4, 5, 6, 7, 8]))
    Hk = int(rng.choice([1, 2, 3]))
    H, D = G * Hk, 128
    S = int(rng.choice([16, 32, 64]))
    window = int(rng.choice([0, 0, int(rng.integers(1, 700))]))
    seqs = []
    for _ in range(int(rng.integers(1, 5))):
        n = int(rng.choice([1, int(rng.integers(2, 40)), int(rng.integers(40, 400))]))
        off = int(rng.choice([0, int(rng.integers(1, 300)), int(rng.integers(300, 3000))]))
        seqs.append((off, n))
    q, kp, vp, bt, sot, pos, want = paged_case(torch.bfloat16, seqs, H, Hk, D, S, window, seed=950 + seed)
    cu, offs = prefill_inputs(seqs)
    max_kv = max(o + n for o, n in seqs) if seed % 2 == 0 else 0
    out = ops().paged_prefill_attention_tc(q, H * D, kp, vp, bt, cu, offs, 1 / math.sqrt(D), window, H, Hk, D,
                                           len(seqs), max(n for _, n in seqs), q.shape[0], max_kv=max_kv)
    ops().check_device_errors()
    close(out, want, torch.bfloat16, what="drawn case %d: %r, %d/%d heads, pages of %d, window %d" % (seed, seqs, H, Hk, S, window))


@pytest.mark.parametrize("far", [0, 500, 1023, 1024, 2900])
def test_prefill_attention_tc_in_runs_finds_one_far_key(far):
    H, Hk, D, S = 8, 2, 128, 16
    seqs = [(2960, 40)]
    q, kp, vp, bt, sot, pos, want = paged_case(torch.bfloat16, seqs, H, Hk, D, S, 0, seed=18, spike=far)
    cu, offs = prefill_inputs(seqs)
    out = ops().paged_prefill_attention_tc(q, H * D, kp, vp, bt, cu, offs, 1 / math.sqrt(D), 0, H, Hk, D, 1, 40, 40, max_kv=3000)
    ops().check_device_errors()
    close(out, want, torch.bfloat16)
    page, off = int(bt[0, far // S]), far % S
    value = vp[page, 0, off].float().cpu().numpy()
    scale = np.abs(value).max()
    assert np.abs(want[-1, :D] - value).max() < 0.03 * scale, "the far key does not decide the plain answer: the case lost its point"
    assert np.abs(f64(out)[-1, :D] - value).max() < 0.04 * scale


# ----------------------------------------------------------------------------
class _NoCalls:
    """A call module that leaves everything to the wrappers in Python."""

    def __getattr__(self, name):
        return lambda *args: None


@pytest.mark.parametrize("rows", [1, 8, 9, 40, 130])
def test_call_module_agrees_with_the_wrappers(rows, monkeypatch):
    """The operations that go through the call module give the bits that their Python wrappers give, and count as launches."""
    o = ops()
    H, Hk, D, S, E = 8, 2, 128, 16, 256
    g = torch.Generator(device=DEV)
    g.manual_seed(rows)
    rnd = lambda *shape: torch.randn(shape, generator=g, device=DEV)
    res, delta, w = rnd(rows, E), rnd(rows, E).bfloat16(), rnd(E)
    wq, wg = rnd((H + 2 * Hk) * D, E).bfloat16(), rnd(512, E).bfloat16()
    qw, kw, inv = rnd(D), rnd(D), torch.rand(D // 2, device=DEV)
    pos = torch.arange(rows, dtype=torch.int32, device=DEV)
    pages = -(-rows // S) + 1
    bt = torch.arange(pages, dtype=torch.int32, device=DEV).view(1, -1)
    cu = torch.tensor([0, rows], dtype=torch.int32, device=DEV)
    zero = torch.zeros(1, dtype=torch.int32, device=DEV)
    some = torch.tensor([rows - 1, 0], dtype=torch.int32, device=DEV)

    def all_of_them():
        r = res.clone()
        kp, vp = torch.zeros(pages, Hk, S, D, device=DEV).bfloat16(), torch.zeros(pages, Hk, S, D, device=DEV).bfloat16()
        n0 = o.launch_count()
        h = o.add_rmsnorm(r, delta, w, 1e-6, torch.bfloat16)
        out = [r, h, o.add_rmsnorm(r, None, w, 1e-6, torch.float32), o.add_rmsnorm(r, delta, w, 1e-6, torch.bfloat16, rows=some)]
        qkv = o.gemm_bf16(h, wq)
        out += [o.gemm_bf16(h, wq, out_dtype=torch.float32), qkv.clone()]
        o.qk_norm_rope_kv(qkv, qw, kw, 1e-6, inv, D, pos, pos, kp, vp, H, Hk, D)
        out += [qkv, kp, vp]
        seq = torch.zeros(rows, dtype=torch.int32, device=DEV)
        out.append(o.paged_decode_attention(qkv, qkv.shape[1], kp, vp, bt, seq, pos, 0.1, 0, H, Hk, D, rows, rows, single_tokens=False))
        out.append(o.paged_prefill_attention_tc(qkv, qkv.shape[1], kp, vp, bt, cu, zero, 0.1, 0, H, Hk, D, 1, rows, rows, max_kv=rows))
        out += [o.gemm_tcgen05(h, wg, gated_activation="silu"), o.gemm_tcgen05(h, wg, pair=True),
                o.gemm_tcgen05(h, wg, activation="relu"), o.gated_act(o.gemm_bf16(h, wg, out_dtype=torch.float32), "silu", 8, torch.bfloat16)]
        o.check_device_errors()
        return out, o.launch_count() - n0

    o._full_precision_sums()
    fast, n_fast = all_of_them()
    monkeypatch.setattr(o, "_CALLS", _NoCalls())
    slow, n_slow = all_of_them()
    assert n_fast == n_slow
    for i, (x, y) in enumerate(zip(fast, slow)):
        assert x.dtype == y.dtype and torch.equal(x, y), i


def test_call_module_leaves_refusals_to_the_wrappers():
    """What a wrapper refuses is refused with its message, whether or not the call module looked at it first."""
    from velox_b200.csrc.ops import KernelError
    o = ops()
    x, w = torch.zeros(4, 64, device=DEV), torch.ones(64, device=DEV)
    with pytest.raises(KernelError, match="weight has 32 elements"):
        o.add_rmsnorm(x, None, w[:32], 1e-6, torch.bfloat16)
    with pytest.raises(KernelError, match="delta must match"):
        o.add_rmsnorm(x, x.bfloat16()[:2], w, 1e-6, torch.bfloat16)
    with pytest.raises(KernelError, match="CUDA tensors"):
        o.add_rmsnorm(x.cpu(), None, w.cpu(), 1e-6, torch.bfloat16)
    with pytest.raises(KernelError, match="norm weight size"):
        o.qk_norm_rope_kv(x.bfloat16(), w[:8], None, 1e-6, None, 0, torch.zeros(4, dtype=torch.int32, device=DEV), None, None, None, 2, 1, 16)
    with pytest.raises(KernelError, match="bfloat16 operands"):
        o.gemm_bf16(x, x)
    with pytest.raises(KernelError, match="K a multiple of 8"):
        o.gemm_tcgen05(x.bfloat16()[:, :60], x.bfloat16()[:, :60])
    with pytest.raises(KernelError, match="even width"):
        o.gated_act(x[:, :63].contiguous(), "silu")


def test_call_module_passes_on_what_a_truth_value_raises():
    with pytest.raises(RuntimeError, match="ambiguous"):
        ops().add_rmsnorm(torch.zeros(4, 64, device=DEV), torch.zeros(4, 64, device=DEV), torch.ones(64, device=DEV), 1e-6, torch.float32,
                          update_residual=torch.ones(2))


@pytest.mark.parametrize("K", [32, 96, 288, 1024, 1280, 2080, 2560])
@pytest.mark.parametrize("variant", [0, 3, 7, 8])
def test_skinny_product_with_batches_that_are_not_whole(K, variant):
    """K that gives a warp no whole batch of chunks, whole ones only, or whole ones and a rest, by every number of warps
    that the sizes choose.  A sum's error is at most K roundings of 2^-24 of the sum of the products' magnitudes."""
    N, M = 272, 5
    g = torch.Generator().manual_seed(K)
    a, w = torch.randn(M, K, generator=g).bfloat16(), torch.randn(N, K, generator=g).bfloat16()
    out = ops().gemm_skinny(a.to(DEV), w.to(DEV), None, torch.float32, variant=variant).cpu().double()
    want, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    assert ((out - want).abs() <= K * 2.0 ** -24 * size).all()
    gated = ops().gemm_skinny(a.to(DEV), w.to(DEV), None, torch.float32, gated_activation="relu", variant=variant).cpu().double()
    t = want.view(M, N // 16, 2, 8)
    ref = (t[:, :, 0].clamp(min=0) * t[:, :, 1]).reshape(M, -1)
    s = size.view(M, N // 16, 2, 8)
    bound = (K + 2) * 2.0 ** -24 * 2 * (s[:, :, 0] * s[:, :, 1]).reshape(M, -1)
    assert ((gated - ref).abs() <= bound).all()


@pytest.mark.parametrize("N", [4736, 4752, 7104, 7120, 9472, 9488, 13312])
@pytest.mark.parametrize("K", [1280, 5120])
def test_skinny_product_where_the_choice_of_warps_turns(N, K):
    """Numbers of tiles around whole rounds of a B200's SMs (two, three and four blocks each), where the choice between four, five and
    eight warps turns.  The bound is the one above."""
    g = torch.Generator().manual_seed(N)
    a, w = torch.randn(3, K, generator=g).bfloat16().to(DEV), torch.randn(N, K, generator=g).bfloat16().to(DEV)
    out = ops().gemm_skinny(a, w, None, torch.float32).double()
    assert ((out - a.double() @ w.double().T).abs() <= K * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)).all()


@pytest.mark.parametrize("columns", [16, 48, 128, 144, 176, 208, 240, 256])
@pytest.mark.parametrize("M,N,K", [(1, 16, 8), (130, 464, 200), (300, 1040, 320)])
def test_gemm_tcgen05_tiles_of_any_width(M, N, K, columns):
    """Tiles whose last 32 columns are half a tile's, tiles wider than the matrix, several tiles a block: the sums that tiles
    of 256 columns give, bit for bit (every sum is formed over k in the same order), gated, plain with a bias and activated."""
    g = torch.Generator().manual_seed(M + columns)
    a, w = torch.randn(M, K, generator=g).bfloat16().to(DEV), torch.randn(N, K, generator=g).bfloat16().to(DEV)
    bias = torch.randn(N, generator=g).to(DEV)
    for more in (dict(gated_activation="silu"), dict(bias=bias), dict(activation="relu2")):
        wide = ops().gemm_tcgen05(a, w, **more)
        assert torch.equal(ops().gemm_tcgen05(a, w, columns=columns, **more), wide), more
    ops().check_device_errors()


@pytest.mark.parametrize("wide", [0, 1, 2, 15, 48, 255, 300, -1])
def test_gemm_tcgen05_takes_any_wide_as_a_truth_value(wide):
    """The C entry point: 0 for tiles of 128 columns, anything else for tiles of 256, the same sums either way."""
    M, N, K = 130, 464, 200
    g = torch.Generator().manual_seed(3)
    a, w = torch.randn(M, K, generator=g).bfloat16().to(DEV), torch.randn(N, K, generator=g).bfloat16().to(DEV)
    out = torch.zeros(M, N, dtype=torch.bfloat16, device=DEV)
    word = ops()._error_word(a.device)
    assert ops().library().vx_gemm_tcgen05(a.data_ptr(), w.data_ptr(), None, out.data_ptr(), M, N, K, K, K, N, 0, 0, wide, word.data_ptr(),
                                           torch.cuda.current_stream().cuda_stream) == 0
    ops().note_bounded_wait()
    ops().check_device_errors()
    assert torch.equal(out, ops().gemm_tcgen05(a, w))


def test_tcgen05_tile_fills_rounds():
    """The choice of tiles stays within what the kernels take."""
    for m in (1, 128, 129, 312, 777, 2048, 40000):
        for n in (16, 512, 6144, 19456, 34816):
            for k in (64, 2048, 2560, 9728):
                pair, columns = ops().tcgen05_tile(m, n, k, torch.device(DEV))
                assert pair == (columns == 0) and columns % 16 == 0 and columns <= 256
