"""The chunked scans hold the states before a window of chunks at a time: whatever the window, the same bits; and how much they hold."""
import pytest
import torch

from mivi_v4_b200.ops import kernels as K

DEV = "cuda:0"


class Scratch:
    def __init__(self):
        self.sizes = {}

    def get(self, name, shape, dtype):
        t = torch.full(tuple(shape), float("nan"), dtype=dtype, device=DEV)
        self.sizes[name] = t.numel() * t.element_size()
        return t


@pytest.mark.parametrize("state_bytes", [4, 1 << 16, 1 << 20, 2 << 20, 16 << 20])
def test_room_is_bounded(state_bytes):
    """However long the step, no more than SCAN_STATES_BYTES (or ten states, where those are more)."""
    for chunks in (1, 2, 7, 8, 9, 65, 769, 1 << 20):
        room = K.scan_room(chunks, state_bytes)
        assert 1 <= room <= chunks
        held = (room + 2 * (room < chunks)) * state_bytes
        assert held <= max(K.SCAN_STATES_BYTES, 10 * state_bytes)


def test_which_steps_are_short():
    """By the chunks one after the other: a sequence's own or, where they do not fit side by side, all heads' and columns'."""
    n = 148 if not torch.cuda.is_available() else K.n_sms()
    few = K.scan_takes_few
    assert few("channel", 320, 1, 320, 8, 128, 256) and not few("channel", 321, 1, 321, 8, 128, 256)
    assert few("head", 192, 1, 192, 1, 128, 16) and not few("head", 193, 1, 193, 1, 128, 16)
    assert few("token", 160, 1, 160, 1, 128, 16) and not few("token", 161, 1, 161, 1, 128, 16)
    assert few("token", 123, 1, 123, 1, 200, 16) and not few("token", 124, 1, 124, 1, 200, 16)
    # 64 sequences of 16 tokens are 64 chunks for each head and 16 columns
    heads = 10 * n // 64
    assert few("channel", 1024, 64, 16, heads, 128, 16) and not few("channel", 1024, 64, 16, heads + 2, 128, 16)
    assert few("channel", 1024, 64, 16, heads + 2, 32, 16)


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


LENS = [[700], [190, 1, 130, 64, 3, 333], [16] * 40]


@pytest.mark.gpu
@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("kind", ["channel", "head", "head with act", "scalar", "scalar with normalizer"])
@pytest.mark.parametrize("heads,dk,dv", [(2, 70, 66), (40, 64, 64)])
def test_same_bits_in_windows(monkeypatch, lens, kind, heads, dk, dv):
    g = torch.Generator(device=DEV).manual_seed(len(lens))
    N, B, cu = sum(lens), len(lens), [0]
    for n in lens:
        cu.append(cu[-1] + n)
    r = lambda *s: torch.randn(*s, generator=g, device=DEV)
    q, k, z, v, m = r(N, heads * dk), r(N, heads * dk), r(N, heads * dk), r(N, heads * dv), r(N, heads)
    log_a, b, decay = -r(N, heads).abs(), r(N, heads).abs(), torch.rand(heads, generator=g, device=DEV)
    norm = kind == "scalar with normalizer"
    state = r(B + 1, heads, dv + int(norm), dk)
    slots = i32([B - i for i in range(B)])
    got = []
    for room in (1 << 30, 1, 2, 3, 10):
        monkeypatch.setattr(K, "scan_room", lambda chunks, state_bytes: min(room, chunks))
        s, out, ws = state.clone(), torch.full((N, heads * dv), float("nan"), device=DEV), Scratch()
        monkeypatch.setattr(K, "scan_takes_few", lambda *a: False)
        if kind.startswith("scalar"):
            K.scalar_scan(q, k, v, log_a, b, s, slots, i32(cu), out, B, heads, dk, dv, m_tok=m if norm else None, q_scale=0.1,
                          max_len=max(lens), ws=ws)
        else:
            how = dict(decay_logits=z, inv_tau=0.125) if kind == "channel" else dict(head_decay=decay)
            K.decay_scan(q, k, v, s, slots, i32(cu), out, B, heads, dk, dv, q_scale=0.1, act=int("act" in kind), max_len=max(lens), ws=ws, **how)
        assert ws.sizes["scan_before"] <= (room + 2) * heads * (dv + norm) * ((dk + 3) & ~3) * 4
        got.append((out, s))
    assert bool(torch.isfinite(got[0][0]).all())
    for out, s in got[1:]:
        assert torch.equal(out, got[0][0]) and torch.equal(s, got[0][1])
