"""The gated delta rule eight tokens at a time (gdr_block_scan_kernel) against the recurrence in 64 bits, beside the scan token by token on
the same inputs and state.  Both are 32-bit sums of the same terms in another order, so their errors are of one size: the blocks' may be
at most twice the scan's (each is a sum of a few dozen roundings; twice is far outside the spread of such sums), plus one ulp of the largest value."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
D, DEV = 128, "cuda"


def library():
    from imp_b200 import capi
    lib = capi.load()
    lib.imp_gdr_block_floats.restype = ctypes.c_int64
    lib.imp_gdr_state_floats.restype = ctypes.c_int64
    return lib


def ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def to_layout(S, blocks):
    """[slots, H, D, Dv] -> per block of 32 columns 16 planes of 256: element (dimension 16 r + i, column c) at plane i, place 8 c + r."""
    n, H, _, Dv = S.shape
    full = torch.zeros(n, H, D, blocks * 32, dtype=S.dtype, device=S.device)
    full[..., :Dv] = S
    return full.view(n, H, 8, 16, blocks, 32).permute(0, 1, 4, 3, 5, 2).contiguous()


def from_layout(L, Dv):
    n, H, blocks = L.shape[:3]
    return L.permute(0, 1, 5, 3, 2, 4).reshape(n, H, D, blocks * 32)[..., :Dv]


def exact(q, k, v, beta, decay, S):
    T, H, Dv = v.shape
    rep = H // q.shape[1]
    q, k = q.double().repeat_interleave(rep, 1), k.double().repeat_interleave(rep, 1)
    v, beta, decay, S, out = v.double(), beta.double(), decay.double(), S.double().clone(), []
    for t in range(T):
        S = S * decay[t, :, None, None]
        u = beta[t, :, None] * (v[t] - torch.einsum("hd,hdv->hv", k[t], S))
        S = S + k[t, :, :, None] * u[:, None]
        out.append(torch.einsum("hd,hdv->hv", q[t], S))
    return torch.stack(out), S


@pytest.mark.parametrize("lengths", [[1], [7], [8], [9], [16, 1, 17], [33, 2, 100], [250]], ids=str)
@pytest.mark.parametrize("G,H,Dv", [(1, 1, 16), (2, 4, 128), (2, 2, 40)])
@pytest.mark.parametrize("keys", ["random", "alike"])    # alike: every token's key nearly the last one's, where the corrections are largest
def test_blocks_against_the_recurrence(lengths, G, H, Dv, keys):
    lib = library()
    g = torch.Generator().manual_seed(sum(lengths) + Dv)
    T, n = sum(lengths), len(lengths)
    q, k = torch.randn(T, G, D, generator=g), torch.randn(T, G, D, generator=g)
    if keys == "alike":
        k = torch.randn(1, G, D, generator=g) + 0.1 * k
    q, k = (q / q.norm(dim=-1, keepdim=True) * D ** -0.5).to(DEV), (k / k.norm(dim=-1, keepdim=True)).to(DEV)
    v = torch.randn(T, H, Dv, generator=g).to(DEV)
    beta, decay = torch.rand(T, H, generator=g).to(DEV), (torch.rand(T, H, generator=g) ** 0.2).to(DEV)
    decay[::13] = 0.0                                     # a state that is forgotten at once
    S0 = torch.randn(n + 1, H, D, Dv, generator=g).to(DEV)
    blocks = (Dv + 31) // 32
    slots = torch.arange(n, 0, -1, dtype=torch.int32, device=DEV)
    starts = [sum(lengths[:i]) for i in range(n + 1)]
    q_start = torch.tensor(starts, dtype=torch.int32, device=DEV)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    got = {}
    for kind in ("scan", "blocks"):
        state = to_layout(S0, blocks)
        assert state[0].numel() == lib.imp_gdr_state_floats(H, D, Dv)
        out = torch.full((T, H, Dv), float("nan"), device=DEV)
        common = (ptr(q), ptr(k), ptr(v), ptr(beta), ptr(decay), ptr(state), ptr(out))
        if kind == "scan":
            rc = lib.imp_gdr_scan_ex(*common, ptr(q_start), ptr(slots), n, G, D, H, Dv, 0, stream)
        else:
            scratch = torch.empty(lib.imp_gdr_block_floats(T, n, H), device=DEV)
            rc = lib.imp_gdr_block_scan(*common, ptr(scratch), ptr(q_start), ptr(slots), n, max(lengths), G, D, H, Dv, stream)
        assert rc == 0
        torch.cuda.synchronize()
        got[kind] = (out, from_layout(state, Dv))
        assert torch.equal(state[0], to_layout(S0, blocks)[0])      # nobody's slot
    for i in range(n):
        a, b, slot = starts[i], starts[i + 1], int(slots[i])
        o, S = exact(q[a:b], k[a:b], v[a:b], beta[a:b], decay[a:b], S0[slot])
        for part, want in ((0, o), (1, S)):
            mine = [got[kind][part][a:b] if part == 0 else got[kind][part][slot] for kind in ("scan", "blocks")]
            err = [float((m.double() - want).norm()) for m in mine]
            assert err[1] <= 2 * err[0] + 2.0 ** -24 * float(want.abs().max()) * want.numel() ** 0.5, (part, i, err)


def test_other_key_sizes_are_declined():
    lib = library()
    t = torch.zeros(4096, device=DEV)
    i = torch.zeros(8, dtype=torch.int32, device=DEV)
    assert lib.imp_gdr_block_scan(*[ptr(t)] * 8, ptr(i), ptr(i), 1, 1, 1, 64, 1, 16, ctypes.c_void_p(0)) == -2
