"""The (token, route) pairs of a batch sorted by expert: tiles, ids outside the layer, experts that another rank holds."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


class Tiles(C.Structure):
    _fields_ = [("n_tiles", C.c_void_p), ("expert", C.c_void_p), ("pairs", C.c_void_p)]


@pytest.mark.parametrize("n_tok,k,n_experts,missing,wrong", [
    (90, 1, 3, [], []),
    (41, 3, 70, [0, 5, 69], []),          # experts of other ranks: their pairs take no part and are no error
    (33, 8, 128, [], [128]),              # the first id behind the layer's experts
    (33, 8, 128, [127], [128, 129, 0xffffffff]),
    (16, 32, 256, list(range(0, 256, 2)), []),
    (512, 32, 256, [], []),
])
def test_tiles(n_tok, k, n_experts, missing, wrong):
    import torch

    from k2t_internal import internal
    launch = internal("launch_expert_tiles", C.c_int, C.c_void_p, C.c_void_p, C.c_uint32, C.c_uint32, C.c_uint32, C.c_uint32, C.c_void_p, C.POINTER(Tiles), C.c_void_p, C.c_bool)
    most = internal("expert_tiles_max", C.c_uint32, C.c_size_t, C.c_uint32)(n_tok * k, n_experts)
    g = torch.Generator().manual_seed(n_tok)
    ids = torch.randint(0, n_experts, (n_tok, 32), generator=g, dtype=torch.int64)
    for i, w in enumerate(wrong):
        ids[3 * i + 1, i % k] = w
    bases = torch.tensor([0 if e in missing else 256 for e in range(n_experts)], dtype=torch.int64, device="cuda")
    d_ids = ids.to(torch.uint32).cuda()
    n, expert, pairs, err = (torch.zeros(c, dtype=torch.int32, device="cuda") for c in (1, most, 32 * most, 1))
    t = Tiles(n.data_ptr(), expert.data_ptr(), pairs.data_ptr())
    assert launch(torch.cuda.current_stream().cuda_stream, d_ids.data_ptr(), n_tok, k, 32, n_experts, bases.data_ptr(), C.byref(t), err.data_ptr(), False) == 0
    torch.cuda.synchronize()
    assert err.item() == (4 if wrong else 0)
    n = n.item()
    assert n <= most
    got = {}
    for e, p in zip(expert[:n].tolist(), pairs.view(most, 32)[:n].tolist()):
        got.setdefault(e, []).append([i for i in p if i != -1])
    want = {}
    for i in range(n_tok * k):
        e = ids[i // k, i % k].item()
        if e < n_experts and e not in missing:
            want.setdefault(e, []).append(i)
    assert {e: sorted(sum(p, [])) for e, p in got.items()} == want
    assert all(len(p) == 32 for e in got for p in got[e][:-1])
