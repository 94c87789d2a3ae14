"""State-space layers: chunked prefill + decode with carried state equals the one-shot result (CPU), and the
CUDA kernels match the fp32 PyTorch forms (GPU)."""

import pytest
import torch

from modular_b200.nn import state_space as ss


def _cu(lens, device="cpu"):
    return torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=device)


def test_mamba_mixer_chunked_matches_one_shot():
    torch.manual_seed(0)
    m = ss.MambaMixer(hidden=32, d_inner=64, d_state=16, d_conv=4)
    lens = [7, 12]
    h = torch.randn(sum(lens), 32)
    full = m(h, _cu(lens))
    # the same two sequences in two chunks each, then the rest token by token
    state = m.alloc_state(4)
    idx = torch.tensor([2, 0], dtype=torch.int32)
    seqs = [h[:7], h[7:]]
    first = [3, 5]
    out = [[], []]
    c1 = torch.cat([seqs[0][:3], seqs[1][:5]])
    y = m(c1, _cu(first), state, idx, torch.tensor([0, 0], dtype=torch.int32))
    out[0].append(y[:3]); out[1].append(y[3:])
    pos = list(first)
    while any(p < l for p, l in zip(pos, lens)):
        live = [i for i in range(2) if pos[i] < lens[i]]
        x = torch.cat([seqs[i][pos[i] : pos[i] + 1] for i in live])
        y = m(x, _cu([1] * len(live)), state, idx[live], torch.ones(len(live), dtype=torch.int32))
        for j, i in enumerate(live):
            out[i].append(y[j : j + 1]); pos[i] += 1
    got = torch.cat([torch.cat(out[0]), torch.cat(out[1])])
    assert torch.allclose(got, full, atol=1e-4, rtol=1e-4)


def test_mamba2_mixer_chunked_matches_one_shot():
    torch.manual_seed(1)
    m = ss.Mamba2Mixer(hidden=32, n_heads=4, head_dim=8, d_state=16, n_groups=2, d_conv=4)
    lens = [9, 4]
    h = torch.randn(sum(lens), 32)
    full = m(h, _cu(lens))
    state = m.alloc_state(2)
    idx = torch.tensor([1, 0], dtype=torch.int32)
    a = m(torch.cat([h[:5], h[9:11]]), _cu([5, 2]), state, idx, torch.zeros(2, dtype=torch.int32))
    b = m(torch.cat([h[5:9], h[11:13]]), _cu([4, 2]), state, idx, torch.ones(2, dtype=torch.int32))
    got = torch.cat([a[:5], b[:4], a[5:], b[4:]])
    assert torch.allclose(got, full, atol=1e-4, rtol=1e-4)


def _rel(a, b):
    a, b = a.float(), b.float()
    return ((a - b).norm() / (b.norm() + 1e-6)).item()


@pytest.mark.gpu
@pytest.mark.parametrize("W", [2, 4])
def test_causal_conv1d_kernel(W):
    torch.manual_seed(2)
    dev = "cuda"
    lens = [1, 33, 7, 128]
    D = 200
    x = torch.randn(sum(lens), D, device=dev, dtype=torch.bfloat16)
    w = (torch.randn(D, W, device=dev) * 0.5).to(torch.bfloat16)
    b = torch.randn(D, device=dev, dtype=torch.bfloat16)
    idx = torch.tensor([3, -1, 0, 1], dtype=torch.int32, device=dev)
    init = torch.tensor([1, 0, 0, 1], dtype=torch.int32, device=dev)
    st = torch.randn(4, D, W - 1, device=dev)
    st_ref = st.clone()
    y = ss.causal_conv1d_varlen(x, w, b, _cu(lens, dev), st, idx, init, True)
    y_ref = ss.causal_conv1d_reference(x, w, b, _cu(lens), st_ref, idx.cpu(), init.cpu(), True)
    assert _rel(y, y_ref) < 1e-2
    assert torch.allclose(st, st_ref, atol=1e-5)


@pytest.mark.gpu
@pytest.mark.parametrize("N", [16, 32])
def test_selective_scan_kernel(N):
    torch.manual_seed(3)
    dev = "cuda"
    lens = [5, 1, 64]
    T, D = sum(lens), 192
    u = torch.randn(T, D, device=dev, dtype=torch.bfloat16)
    delta = (torch.randn(T, D, device=dev) * 0.5).to(torch.bfloat16)
    A = -torch.rand(D, N, device=dev) - 0.1
    B = torch.randn(T, N, device=dev, dtype=torch.bfloat16)
    C = torch.randn(T, N, device=dev, dtype=torch.bfloat16)
    Dk = torch.randn(D, device=dev)
    z = torch.randn(T, D, device=dev, dtype=torch.bfloat16)
    bias = torch.randn(D, device=dev) * 0.1
    idx = torch.tensor([1, 0, -1], dtype=torch.int32, device=dev)
    init = torch.tensor([0, 1, 0], dtype=torch.int32, device=dev)
    st = torch.randn(2, D, N, device=dev)
    st_ref = st.clone()
    y = ss.selective_scan_varlen(u, delta, A, B, C, Dk, z, bias, _cu(lens, dev), st, idx, init, True)
    y_ref = ss.selective_scan_reference(u, delta, A, B, C, Dk, z, bias, _cu(lens), st_ref, idx.cpu(), init.cpu(), True)
    assert _rel(y, y_ref) < 1e-2
    assert _rel(st, st_ref) < 1e-3


@pytest.mark.gpu
@pytest.mark.parametrize("H,P,N,G", [(4, 64, 128, 1), (6, 32, 64, 2), (2, 128, 16, 2)])
def test_ssd_scan_kernel(H, P, N, G):
    torch.manual_seed(4)
    dev = "cuda"
    lens = [3, 40, 1]
    T = sum(lens)
    x = torch.randn(T, H, P, device=dev, dtype=torch.bfloat16)
    dt = (torch.randn(T, H, device=dev) * 0.5).to(torch.bfloat16)
    A = -torch.rand(H, device=dev) - 0.1
    B = (torch.randn(T, G, N, device=dev) * 0.3).to(torch.bfloat16)
    C = (torch.randn(T, G, N, device=dev) * 0.3).to(torch.bfloat16)
    Dk = torch.randn(H, device=dev)
    bias = torch.randn(H, device=dev) * 0.1
    idx = torch.tensor([0, 2, 1], dtype=torch.int32, device=dev)
    init = torch.tensor([1, 0, 1], dtype=torch.int32, device=dev)
    st = torch.randn(3, H, P, N, device=dev) * 0.2
    st_ref = st.clone()
    y = ss.ssd_scan_varlen(x, dt, A, B, C, Dk, bias, _cu(lens, dev), st, idx, init, True)
    y_ref = ss.ssd_scan_reference(x, dt, A, B, C, Dk, bias, _cu(lens), st_ref, idx.cpu(), init.cpu(), True)
    assert _rel(y, y_ref) < 1e-2
    assert _rel(st, st_ref) < 1e-3


def _strided(t, lead=8):
    """The same values as rows of a wider tensor (another distance between rows, another first column)."""
    wide = torch.zeros(t.shape[0], lead + t[0].numel() + 8, device=t.device, dtype=t.dtype)
    wide[:, lead: lead + t[0].numel()] = t.flatten(1)
    return wide[:, lead: lead + t[0].numel()].view(t.shape)


EDGES = [1, 63, 0, 64, 65, 2, 130, 31, 33]        # around tiles of 16, 32 and 64 tokens, an empty sequence among them


def _state_args(dev):
    idx = torch.tensor([3, -1, 0, 1, 2, 4, 8, 5, 6], dtype=torch.int32, device=dev)
    init = torch.tensor([1, 0, 0, 1, 0, 1, 1, 1, 0], dtype=torch.int32, device=dev)
    return idx, init


@pytest.mark.gpu
@pytest.mark.parametrize("W,D,lead", [(4, 1032, 8), (2, 64, 16), (8, 8, 8), (3, 24, 1), (4, 13, 3)])
def test_conv_tiles(W, D, lead):
    """Aligned rows (8 channels a thread) and rows that are not (1)."""
    torch.manual_seed(5)
    dev = "cuda"
    idx, init = _state_args(dev)
    x = _strided(torch.randn(sum(EDGES), D, device=dev).to(torch.bfloat16), lead)
    w, b = (torch.randn(D, W, device=dev) * 0.5).to(torch.bfloat16), torch.randn(D, device=dev).to(torch.bfloat16)
    st = torch.randn(9, D, W - 1, device=dev)
    ref = st.clone()
    y = ss.causal_conv1d_varlen(x, w, b, _cu(EDGES, dev), st, idx, init, True)
    want = ss.causal_conv1d_reference(x, w, b, _cu(EDGES), ref, idx.cpu(), init.cpu(), True)
    assert _rel(y, want) < 2 ** -8                 # one rounding to bf16 on either side
    assert torch.equal(st, ref)                    # the state is a copy of inputs


@pytest.mark.gpu
@pytest.mark.parametrize("N,D,lead", [(16, 40, 8), (8, 32, 8), (32, 72, 8), (16, 37, 8), (16, 64, 1)])
def test_selective_scan_tiles(N, D, lead):
    torch.manual_seed(6)
    dev, T = "cuda", sum(EDGES)
    idx, init = _state_args(dev)
    bf = lambda *s, k=1.0: (torch.randn(*s, device=dev) * k).to(torch.bfloat16)
    u, delta, z, B, C = bf(T, D), bf(T, D, k=0.5), _strided(bf(T, D), lead), _strided(bf(T, N), lead), _strided(bf(T, N), lead)
    A, Dk, bias = -torch.rand(D, N, device=dev) * 4 - 0.1, torch.randn(D, device=dev), torch.randn(D, device=dev) * 0.1
    st = torch.randn(9, D, N, device=dev)
    ref = st.clone()
    y = ss.selective_scan_varlen(u, delta, A, B, C, Dk, z, bias, _cu(EDGES, dev), st, idx, init, True)
    want = ss.selective_scan_reference(u, delta, A, B, C, Dk, z, bias, _cu(EDGES), ref, idx.cpu(), init.cpu(), True)
    assert _rel(y, want) < 2 ** -8
    assert _rel(st, ref) < 1e-5                    # fp32: 2 ulp of ex2.approx per step over the state's memory of a few steps


@pytest.mark.gpu
@pytest.mark.parametrize("N,D,lead", [(16, 2048, 8), (8, 2056, 8), (32, 2048, 8), (16, 2051, 1)])
def test_selective_scan_is_the_same_in_any_batch(N, D, lead):
    """Batches of many channels give a channel four lanes, single sequences eight: the states are the same, bit for bit, and
    outputs differ by the order of a sum over N states (a rounding to bf16 apart)."""
    torch.manual_seed(16)
    dev, lens = "cuda", [1, 7, 8, 9, 31, 32, 33, 70]
    T, cu = sum(lens), _cu(lens, dev)
    bf = lambda *s, k=1.0: (torch.randn(*s, device=dev) * k).to(torch.bfloat16)
    u, delta, z, B, C = bf(T, D), bf(T, D, k=0.5), _strided(bf(T, D), lead), _strided(bf(T, N), lead), _strided(bf(T, N), lead)
    A, Dk, bias = -torch.rand(D, N, device=dev) * 4 - 0.1, torch.randn(D, device=dev), torch.randn(D, device=dev) * 0.1
    idx = torch.tensor([5, 0, -1, 3, 1, 6, 2, 7], dtype=torch.int32, device=dev)
    init = torch.tensor([1, 0, 0, 1, 0, 1, 0, 1], dtype=torch.int32, device=dev)
    st = torch.randn(8, D, N, device=dev)
    one = st.clone()
    y = ss.selective_scan_varlen(u, delta, A, B, C, Dk, z, bias, cu, st, idx, init, True)
    for i, n in enumerate(lens):
        r = slice(sum(lens[:i]), sum(lens[:i]) + n)
        w = ss.selective_scan_varlen(u[r], delta[r], A, B[r], C[r], Dk, z[r], bias, _cu([n], dev), one, idx[i: i + 1], init[i: i + 1], True)
        assert _rel(y[r], w) < 2 ** -9
    assert torch.equal(st, one)


@pytest.mark.gpu
@pytest.mark.parametrize("lens", [[31] * 15 + [47], [31] * 16])
def test_selective_scan_of_32_states_is_the_same_in_any_batch(lens):
    """Four lanes a channel from 32 tokens a sequence on, eight below and for single sequences: the same states, bit for bit."""
    torch.manual_seed(20)
    dev, D, N, T = "cuda", 1024, 32, sum(lens)
    bf = lambda *s, k=1.0: (torch.randn(*s, device=dev) * k).to(torch.bfloat16)
    u, delta, z, B, C = bf(T, D), bf(T, D, k=0.5), bf(T, D), bf(T, N), bf(T, N)
    A, Dk, bias = -torch.rand(D, N, device=dev) * 4 - 0.1, torch.randn(D, device=dev), torch.randn(D, device=dev) * 0.1
    idx, init = torch.arange(16, dtype=torch.int32, device=dev), torch.ones(16, dtype=torch.int32, device=dev)
    st = torch.randn(16, D, N, device=dev)
    one = st.clone()
    y = ss.selective_scan_varlen(u, delta, A, B, C, Dk, z, bias, _cu(lens, dev), st, idx, init, True)
    for i, n in enumerate(lens):
        r = slice(sum(lens[:i]), sum(lens[:i]) + n)
        w = ss.selective_scan_varlen(u[r], delta[r], A, B[r], C[r], Dk, z[r], bias, _cu([n], dev), one, idx[i: i + 1], init[i: i + 1], True)
        assert _rel(y[r], w) < 2 ** -9                 # the order of a sum over 32 states, then a rounding to bf16
    assert torch.equal(st, one)


@pytest.mark.gpu
@pytest.mark.parametrize("H,P,N,G,A0", [(4, 64, 128, 1, 1.0), (6, 32, 64, 2, 16.0), (2, 128, 16, 2, 0.1), (3, 8, 24, 1, 1.0), (2, 16, 40, 2, 4.0),
                                        (2, 4, 16, 1, 1.0), (2, 64, 136, 1, 1.0)])
def test_ssd_chunks(H, P, N, G, A0):
    """Chunks of 64 on the tensor cores; the last two sizes stay with the token walk."""
    torch.manual_seed(7)
    dev, T = "cuda", sum(EDGES)
    idx, init = _state_args(dev)
    bf = lambda *s, k=1.0: (torch.randn(*s, device=dev) * k).to(torch.bfloat16)
    x, dt, B, C = _strided(bf(T, H, P)), _strided(bf(T, H, k=0.5), 1), _strided(bf(T, G, N, k=0.3)), _strided(bf(T, G, N, k=0.3))
    A, Dk, bias = -A0 * (torch.rand(H, device=dev) + 0.1), torch.randn(H, device=dev), torch.randn(H, device=dev) * 0.1
    st = torch.randn(9, H, P, N, device=dev)
    ref = st.clone()
    y = ss.ssd_scan_varlen(x, dt, A, B, C, Dk, bias, _cu(EDGES, dev), st, idx, init, True)
    want = ss.ssd_scan_reference(x, dt, A, B, C, Dk, bias, _cu(EDGES), ref, idx.cpu(), init.cpu(), True)
    assert _rel(y, want) < 2 ** -8
    assert _rel(st, ref) < 1e-5                    # three-part operands keep 24 bits; a sum of up to 130 fp32 terms and powers


@pytest.mark.gpu
@pytest.mark.parametrize("D", [8, 2048, 2056, 5120, 16384, 100])
def test_gated_rms_norm(D):
    torch.manual_seed(8)
    y, z = (torch.randn(5, D, device="cuda").to(torch.bfloat16) for _ in range(2))
    w, z = torch.randn(D, device="cuda").to(torch.bfloat16), _strided(z)
    g = y.double() * z.double() / (1 + torch.exp(-z.double()))
    want = g * torch.rsqrt(g.pow(2).mean(-1, keepdim=True) + 1e-5) * w.double()
    assert _rel(ss.gated_rms_norm(y, z, w, 1e-5), want) < 2 ** -8


@pytest.mark.gpu
@pytest.mark.parametrize("H,P,N", [(1, 64, 16), (1, 4, 16), (4, 1, 8), (4, 32, 1)])
def test_strides_of_single_elements(H, P, N):
    """Dimensions of one element may have any stride: one head, one group, one value, one channel."""
    torch.manual_seed(9)
    dev, lens = "cuda", [40, 1]
    T, cu = sum(lens), _cu(lens, dev)
    bf = lambda *s, k=1.0: (torch.randn(*s, device=dev) * k).to(torch.bfloat16)
    loose = lambda t: torch.as_strided(t, t.shape, [st if n != 1 else 7777 for st, n in zip(t.stride(), t.shape)])
    x, dt, B, C = bf(T, H, P), bf(T, H, k=0.5), bf(T, 1, N), bf(T, 1, N)
    A = -torch.rand(H, device=dev) - 0.1
    want = ss.ssd_scan_varlen(x, dt, A, B, C, None, None, cu)
    assert torch.equal(ss.ssd_scan_varlen(loose(x), loose(dt), A, loose(B), loose(C), None, None, cu), want)
    if H == 1:
        assert torch.equal(ss.ssd_scan_varlen(x, dt.flatten(), A, B, C, None, None, cu), want)
    u, z, b, c = bf(T, 1), bf(T, 1), bf(T, 8), bf(T, 8)
    a = -torch.rand(1, 8, device=dev)
    want = ss.selective_scan_varlen(u, u, a, b, c, None, z, None, cu)
    assert torch.equal(ss.selective_scan_varlen(u, u, a, b, c, None, loose(z), None, cu), want)
    assert torch.equal(ss.selective_scan_varlen(u, u, a, b.unsqueeze(2), c, None, z.unsqueeze(2), None, cu), want)


@pytest.mark.gpu
@pytest.mark.parametrize("lens,H,P,N,A0", [([4000, 1, 800], 4, 64, 128, 1.0), ([1537], 3, 72, 64, 0.05), ([512, 0, 4608, 1025], 2, 32, 24, 0.01),
                                             ([10000], 1, 16, 8, 0.003)])
def test_ssd_segments(lens, H, P, N, A0):
    """Long prompts in segments of 512 tokens and more, ragged, beside short ones: the same as in portions of 500 tokens that are walked whole."""
    torch.manual_seed(17)
    dev, T, B_ = "cuda", sum(lens), len(lens)
    bf = lambda *s, k=1.0: (torch.randn(*s, device=dev) * k).to(torch.bfloat16)
    x, dt, B, C = bf(T, H, P), bf(T, H, k=0.5), bf(T, 1, N), bf(T, 1, N)
    A, Dk, bias = -torch.rand(H, device=dev) * A0 - 1e-3, torch.randn(H, device=dev), torch.randn(H, device=dev) * 0.1
    idx = torch.tensor([3, -1, 0, 2][:B_], dtype=torch.int32, device=dev)
    init = torch.tensor([1, 0, 0, 1][:B_], dtype=torch.int32, device=dev)
    start = torch.randn(5, H, P, N, device=dev)
    st = start.clone()
    y = ss.ssd_scan_varlen(x, dt, A, B, C, Dk, bias, _cu(lens, dev), st, idx, init, True)
    for i, n in enumerate(lens):
        if n == 0:
            continue
        one, slot = start.clone(), max(int(idx[i]), 0)
        keep = torch.tensor([slot if int(idx[i]) >= 0 else 4], dtype=torch.int32, device=dev)      # a slot of its own for the one without
        want = []
        for c in range(0, n, 500):
            r = slice(sum(lens[:i]) + c, sum(lens[:i]) + min(c + 500, n))
            want.append(ss.ssd_scan_varlen(x[r], dt[r], A, B[r], C[r], Dk, bias, _cu([r.stop - r.start], dev), one, keep,
                                           init[i: i + 1] if c == 0 else torch.ones(1, dtype=torch.int32, device=dev), True))
        assert _rel(y[sum(lens[:i]): sum(lens[:i]) + n], torch.cat(want)) < 2 ** -8          # a rounding to bf16 on either side
        if int(idx[i]) >= 0:
            assert _rel(st[slot], one[slot]) < 1e-5        # fp32 sums over the state's memory, cut at other tokens
    assert torch.equal(st[1], start[1]) and torch.equal(st[4], start[4])


@pytest.mark.gpu
@pytest.mark.parametrize("lens,H,N", [([4097, 4097], 80, 128), ([513, 3585], 20, 24), ([4097], 3, 64)])
def test_ssd_segments_continue_kept_states(lens, H, N):
    """Every sequence goes on from a kept state that decays slowly and is far from the new one, its last segment is one token (the first to
    end), and the first case has more CTAs than the chip holds at once: all segments start from the kept state, none from the new one."""
    torch.manual_seed(18)
    dev, T, P = "cuda", sum(lens), 64
    bf = lambda *s, k=1.0: (torch.randn(*s, device=dev) * k).to(torch.bfloat16)
    x, dt, B, C = bf(T, H, P), bf(T, H, k=0.5), bf(T, 1, N), bf(T, 1, N)
    A, bias = -torch.rand(H, device=dev) * 1e-3 - 1e-3, torch.randn(H, device=dev) * 0.1
    idx = torch.tensor([2, 0][: len(lens)], dtype=torch.int32, device=dev)
    one = torch.ones(len(lens), dtype=torch.int32, device=dev)
    st = torch.randn(3, H, P, N, device=dev) * 10
    want_st, want = st.clone(), []
    y = ss.ssd_scan_varlen(x, dt, A, B, C, None, bias, _cu(lens, dev), st, idx, one, True)
    for i, n in enumerate(lens):
        for c in range(0, n, 500):                     # portions that are walked whole
            r = slice(sum(lens[:i]) + c, sum(lens[:i]) + min(c + 500, n))
            want.append(ss.ssd_scan_varlen(x[r], dt[r], A, B[r], C[r], None, bias, _cu([r.stop - r.start], dev), want_st, idx[i: i + 1], one[:1], True))
    want = torch.cat(want)
    for r in range(0, T, 256):                         # a stretch by itself: one wrong segment is a small part of the whole
        assert _rel(y[r: r + 256], want[r: r + 256]) < 2 ** -8          # a rounding to bf16 on either side
    assert _rel(st, want_st) < 1e-5                    # fp32 sums over the state's memory, cut at other tokens


@pytest.mark.gpu
@pytest.mark.parametrize("lens,H,N", [([4097], 110, 128), ([4097, 4097], 80, 24)])
def test_ssd_segments_on_a_full_chip(lens, H, N):
    """The most heads that one sequence, and narrow states of two, are cut into segments for: more CTAs than the chip holds at once."""
    test_ssd_segments_continue_kept_states(lens, H, N)


@pytest.mark.gpu
@pytest.mark.parametrize("lens", [[0, 2000, 1700], [1700, 3000]])
def test_ssd_segments_leave_rows_before_the_first_sequence(lens):
    """Sequences that begin some segments into the rows: nobody walks the rows before them, and an empty one keeps its state."""
    torch.manual_seed(19)
    dev, lead, H, P, N = "cuda", 1300, 3, 64, 64
    T = lead + sum(lens)
    bf = lambda *s, k=1.0: (torch.randn(*s, device=dev) * k).to(torch.bfloat16)
    x, dt, B, C = bf(T, H, P), bf(T, H, k=0.5), bf(T, 1, N), bf(T, 1, N)
    A = -torch.rand(H, device=dev) * 1e-2 - 1e-3
    idx, one = torch.arange(len(lens), dtype=torch.int32, device=dev), torch.ones(len(lens), dtype=torch.int32, device=dev)
    st = torch.randn(len(lens), H, P, N, device=dev)
    start, want = st.clone(), st.clone()
    y = torch.full_like(x, 7.0)
    from modular_b200._native import lib
    lib().ssd_scan_varlen(x, dt, A, B, C, None, None, y, st, _cu([lead, *lens], dev)[1:].contiguous(), idx, one, True)
    w = ss.ssd_scan_varlen(x[lead:], dt[lead:], A, B[lead:], C[lead:], None, None, _cu(lens, dev), want, idx, one, True)
    assert (y[:lead] == 7.0).all()
    assert _rel(y[lead:], w) < 2 ** -8 and _rel(st, want) < 1e-5          # segments begin at other tokens
    for i, n in enumerate(lens):
        assert n > 0 or torch.equal(st[i], start[i])


@pytest.mark.gpu
def test_silu_of_large_negative_inputs():
    """silu(x) down to where it leaves bf16's normal numbers: 1 + exp(-x) is above 2^126 from -87.4 on, where a fast division gives zero."""
    dev = "cuda"
    v = torch.tensor([-88.5, -88.0, -87.5, -87.0, -60.0, -20.0, -1.0, 0.5], device=dev).bfloat16().repeat(20, 1).contiguous()
    want = (v.double() * torch.sigmoid(v.double()))
    close = lambda a, b: torch.allclose(a.double(), b, rtol=2 ** -7, atol=0)          # __expf of 88 is good to 2^-15, then a rounding to bf16
    w = torch.zeros(8, 4, device=dev, dtype=torch.bfloat16)
    w[:, 3] = 1
    assert close(ss.causal_conv1d_varlen(v, w, None, _cu([20], dev)), want)
    y, one = torch.full_like(v, 2.0), torch.ones(8, device=dev, dtype=torch.bfloat16)
    g = 2 * want
    assert close(ss.gated_rms_norm(y, v, one, 1e-6), g * (g.square().mean(1, keepdim=True) + 1e-6).rsqrt())
    zero = torch.zeros_like(v)
    scan = ss.selective_scan_varlen(one.expand(20, 8).contiguous(), zero, -torch.ones(8, 8, device=dev), zero, zero, torch.ones(8, device=dev), v, None, _cu([20], dev))
    assert close(scan, want)


@pytest.mark.gpu
def test_ssd_special_inputs_stay_causal():
    """An infinite or NaN input of a prompt changes its own row of the state from its token on, and nothing before it."""
    torch.manual_seed(10)
    dev, lens, (H, P, N) = "cuda", [150, 64, 70], (3, 32, 16)
    T = sum(lens)
    bf = lambda *s, k=1.0: (torch.randn(*s, device=dev) * k).to(torch.bfloat16)
    x, dt, B, C = bf(T, H, P), bf(T, H, k=0.5), bf(T, 1, N, k=0.3), bf(T, 1, N, k=0.3)
    x[77, 1, 3], x[5, 0, 8], x[149, 2, 0], x[150 + 63, 2, 31] = float("inf"), float("nan"), -float("inf"), float("nan")
    A, bias, st = -torch.rand(H, device=dev) - 0.1, torch.randn(H, device=dev) * 0.1, torch.randn(3, H, P, N, device=dev)
    ref, idx, init = st.clone(), torch.arange(3, dtype=torch.int32, device=dev), torch.ones(3, dtype=torch.int32, device=dev)
    y = ss.ssd_scan_varlen(x, dt, A, B, C, None, bias, _cu(lens, dev), st, idx, init, True).cpu()
    want = ss.ssd_scan_reference(x.cpu(), dt.cpu(), A.cpu(), B.cpu(), C.cpu(), None, bias.cpu(), _cu(lens), ref.cpu(), idx.cpu(), init.cpu(), True)
    ok = torch.isfinite(want)
    assert torch.equal(torch.isfinite(y), ok) and not ok.all()
    assert _rel(y[ok], want[ok]) < 2 ** -8


@pytest.mark.gpu
def test_ssd_decays_of_many_octaves():
    """Every eleventh token all but clears the state (2^-94000 and less): what follows it keeps its own, small decays."""
    torch.manual_seed(11)
    dev, T, (H, P, N) = "cuda", 200, (4, 32, 64)
    bf = lambda *s, k=1.0: (torch.randn(*s, device=dev) * k).to(torch.bfloat16)
    dt = torch.rand(T, H, device=dev) * 2.0 ** -15
    dt[::11] = 2.0 + torch.rand(H, device=dev)
    dt = dt.to(torch.bfloat16)
    x, B, C, A = bf(T, H, P), bf(T, 1, N, k=0.3), bf(T, 1, N, k=0.3), torch.full((H,), -2.0 ** 15, device=dev)
    y = ss.ssd_scan_varlen(x, dt, A, B, C, None, None, _cu([T], dev), dt_softplus=False)
    want = ss.ssd_scan_reference(x.cpu().float(), dt.cpu(), A.cpu(), B.cpu(), C.cpu(), None, None, _cu([T]), dt_softplus=False)
    assert _rel(y.cpu(), want) < 2 ** -8                 # one rounding to bf16


@pytest.mark.gpu
def test_decays_of_zero():
    """Rates so large that a decay is zero (A = -exp(A_log) of minus infinity, sums beyond the largest float): each token alone is left."""
    torch.manual_seed(12)
    dev, T, (H, P, N) = "cuda", 133, (3, 32, 16)
    bf = lambda *s, k=1.0: (torch.randn(*s, device=dev) * k).to(torch.bfloat16)
    A = torch.tensor([-float("inf"), -3e38, -0.5], device=dev)
    x, dt, B, C, st = bf(T, H, P), bf(T, H, k=0.3), bf(T, 1, N, k=0.3), bf(T, 1, N, k=0.3), torch.randn(1, H, P, N, device=dev)
    ref, idx, init = st.clone().cpu(), torch.zeros(1, dtype=torch.int32, device=dev), torch.ones(1, dtype=torch.int32, device=dev)
    y = ss.ssd_scan_varlen(x, dt, A, B, C, None, None, _cu([T], dev), st, idx, init, True)
    want = ss.ssd_scan_reference(x.cpu().float(), dt.cpu(), A.cpu(), B.cpu(), C.cpu(), None, None, _cu([T]), ref, idx.cpu(), init.cpu(), True)
    for h in range(H):
        assert _rel(y[:, h].cpu(), want[:, h]) < 2 ** -8 and _rel(st[0, h].cpu(), ref[0, h]) < 1e-5, h
    D = 40
    u, delta, b, c = bf(T, D), bf(T, D, k=0.3), bf(T, N, k=0.3), bf(T, N, k=0.3)
    a = -torch.rand(D, N, device=dev) - 0.1
    a[::3], a[1, 2] = -float("inf"), -3e38
    got = ss.selective_scan_varlen(u, delta, a, b, c, None, None, None, _cu([T], dev))
    want = ss.selective_scan_reference(u.cpu().float(), delta.cpu(), a.cpu(), b.cpu(), c.cpu(), None, None, None, _cu([T]))
    assert _rel(got.cpu(), want) < 2 ** -8
