"""The matrix memory's n and m are read by every block of a request's head and written once: a step of many requests, whose
blocks do not all run at once, gives the same bits every time, and those of each request alone."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def i32(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("S,H,N,dv,tokens", [(48, 16, 128, 128, 1), (96, 8, 64, 120, 2), (3, 4, 40, 15, 3)])
def test_a_step_of_many_requests_repeats_itself(S, H, N, dv, tokens):
    from photon_infer_b200.kernels import ops
    g = torch.Generator().manual_seed(S + dv)
    T = S * tokens
    q, k = (torch.randn(T, H * N, generator=g).to(DEV) for _ in range(2))
    v = torch.randn(T, H * dv, generator=g).to(DEV)
    gates = 2.0 * torch.randn(T, 2 * H, generator=g).to(DEV)
    p0, p1 = (0.5 * torch.randn(H, generator=g).to(DEV) for _ in range(2))
    start = 0.3 * torch.randn(S, H * N * dv + H * N + H, generator=g).to(DEV)

    def step(first, last):
        t0, t1 = first * tokens, last * tokens
        state = start.clone()
        out = torch.empty(t1 - t0, H * dv, device=DEV)
        err = torch.zeros(4, dtype=torch.int32, device=DEV)
        ops.linrec("matrix_memory", q[t0:t1], k[t0:t1], v[t0:t1], gates[t0:t1, :H], gates[t0:t1, H:], p0, p1, None, 6.0, N ** -0.5,
                   i32(list(range(0, t1 - t0 + 1, tokens))), i32(list(range(first, last))), state, out, last - first, H, H, N, dv, err)
        assert err.cpu().tolist()[0] == 0
        return out, state

    # a request alone: all of its blocks run at once
    alone = [step(s, s + 1) for s in range(S)]
    want = torch.cat([o for o, _ in alone])
    want_state = torch.stack([st[s] for s, (_, st) in enumerate(alone)])
    for _ in range(8):
        out, state = step(0, S)
        assert torch.equal(out, want)
        assert torch.equal(state, want_state)
