"""Window attention of prompts (bf16) by itself: the launch against 64-bit attention over the rows that it reads, key by key, its bits under cuts of a
prompt, and what a value that is not finite reaches."""
import ctypes as C

import numpy as np
import pytest

from k2t_internal import internal

pytestmark = pytest.mark.gpu


class Act(C.Structure):
    _fields_ = [("p", C.c_void_p), ("ld", C.c_uint32)]


class Ring(C.Structure):
    _fields_ = [("window", C.c_uint32), ("sinks", C.c_uint32), ("ring_len", C.c_uint32)]


class Args(C.Structure):
    _fields_ = [(n, C.c_size_t if n == "qkv_stride" else C.c_void_p) for n in "qkv qkv_stride q_norm k_norm head_scale head_slope k_cache v_cache q pos".split()] + [
        (n, C.c_uint32) for n in "n_q n_kv dim vdim row".split()] + [("ring", Ring), ("eps", C.c_float), ("out", Act), ("err_flag", C.c_void_p), ("ctx_bound", C.c_uint32)]


class Layer:
    """Device rows of one attention layer, and its launches."""

    def __init__(self, heads, kv, dim, vdim, window, ring_len, scale=1.0, slope=0.0, seed=0):
        import torch
        self.torch, self.rng = torch, np.random.default_rng(seed)
        self.H, self.G, self.dim, self.vdim, self.window, self.ring_len = heads, kv, dim, vdim, window, ring_len
        self.row = internal("window_attn_row", C.c_uint32, C.c_uint32, C.c_uint32)(dim, vdim)
        self.k, self.v = (torch.zeros(kv, ring_len, self.row, dtype=torch.bfloat16, device="cuda") for _ in "kv")
        self.ones, self.scale = torch.ones(dim, device="cuda"), torch.from_numpy((scale * dim ** -0.5 * self.rng.uniform(0.5, 1.5, heads)).astype(np.float32)).cuda()
        self.slope = torch.from_numpy((slope * self.rng.uniform(0.5, 1.5, heads)).astype(np.float32)).cuda()

    def inputs(self, n):
        """[n][queries, keys, values] on the host."""
        return self.rng.standard_normal((n, self.H * self.dim + self.G * (self.dim + self.vdim))).astype(np.float32)

    def values(self, qkv):
        """The values of `inputs`, [n][G][vdim]."""
        return qkv[:, -self.G * self.vdim:].reshape(len(qkv), self.G, self.vdim)

    def run(self, qkv, pos):
        """Rows `pos` .. as one batch: the outputs [n][H][vdim] (bf16 values), and the queries [n][H][dim] as the kernel reads them."""
        torch, n = self.torch, len(qkv)
        x = torch.from_numpy(qkv).cuda()
        q = torch.full((n, self.H, self.row), 9.0, dtype=torch.bfloat16, device="cuda")
        at, err, ld = torch.tensor([pos], dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda"), (n + 7) // 8 * 8
        cols = self.H * self.vdim
        out = torch.full(((cols + 63) // 64, ld, 64), -3.0, dtype=torch.bfloat16, device="cuda")
        a = Args(x.data_ptr(), x.shape[1], self.ones.data_ptr(), self.ones.data_ptr(), self.scale.data_ptr(), self.slope.data_ptr(), self.k.data_ptr(), self.v.data_ptr(), q.data_ptr(),
                 at.data_ptr(), self.H, self.G, self.dim, self.vdim, self.row, Ring(self.window, 0, self.ring_len), 1e-6, Act(out.data_ptr(), ld), err.data_ptr(), pos + n)
        launches = C.c_uint32()
        launch = internal("launch_window_attention", C.c_int, C.c_void_p, C.c_bool, C.POINTER(Args), C.c_uint32, C.c_int, C.POINTER(C.c_uint32), C.c_bool)
        assert launch(torch.cuda.current_stream().cuda_stream, False, C.byref(a), n, 148, C.byref(launches), False) == 0
        torch.cuda.synchronize()
        assert err.item() == 0
        # panels of 64 columns, chunk c of token t at c ^ (t & 7)
        chunk = torch.arange(8, device="cuda").view(1, 8) ^ (torch.arange(ld, device="cuda").view(ld, 1) & 7)
        o = out.view(-1, ld, 8, 8).gather(2, chunk.view(1, ld, 8, 1).expand(out.shape[0], ld, 8, 8)).reshape(-1, ld, 64).permute(1, 0, 2).reshape(ld, -1)
        assert (o[n:] == -3).all() and (o[:, cols:] == -3).all()
        return o[:n, :cols].float().cpu().numpy().reshape(n, self.H, self.vdim), q.float().cpu().numpy()[:, :, :self.dim]

    def exact(self, q, pos):
        """64-bit attention of the batch's queries over the cached rows: outputs, and the sums of weights times |values|."""
        n = len(q)
        seen = np.arange(max(0, pos + 1 - (self.window or pos + 1)), pos + n)
        k, v = (c[:, seen % self.ring_len].float().cpu().numpy().astype(np.float64) for c in (self.k, self.v))
        out, size = np.empty((n, self.H, self.vdim)), np.empty((n, self.H, self.vdim))
        away = (pos + np.arange(n))[:, None] - seen[None]
        hide = (away < 0) | (away >= self.window if self.window else False)
        sc, sl = self.scale.cpu().numpy().astype(np.float64), self.slope.cpu().numpy().astype(np.float64)
        for h in range(self.H):
            g = h // (self.H // self.G)
            s = (q[:, h].astype(np.float64) @ k[g, :, :self.dim].T) * sc[h] - sl[h] * away
            s[hide] = -np.inf
            w = np.exp(s - s.max(1, keepdims=True))
            w /= w.sum(1, keepdims=True)
            out[:, h], size[:, h] = w @ v[g, :, :self.vdim], w @ np.abs(v[g, :, :self.vdim])
        return out, size


# heads, kv heads, dim, vdim, window, portions: every head size, both tile heights, groups that end a tile inside a token, windows inside a tile
SHAPES = [(4, 1, 32, 32, 0, [2, 300]), (4, 1, 64, 64, 0, [32]), (6, 2, 128, 128, 0, [33]), (8, 1, 256, 256, 7, [20, 12, 31]), (4, 2, 64, 64, 0, [3, 9, 140]), (3, 1, 96, 80, 100, [129, 42]), (8, 2, 128, 128, 0, [255, 2, 600]), (8, 2, 128, 120, 40, [200, 131]), (2, 2, 128, 128, 17, [128, 129]),
          (5, 1, 192, 192, 100, [27, 150]), (2, 2, 192, 130, 0, [64, 65, 200]), (1, 1, 256, 256, 0, [16, 17, 300]), (2, 2, 256, 250, 9, [128, 130]), (6, 2, 128, 128, 900, [700, 1300])]
# One rounding of a weight and one of the result to bf16 (8 bits: 2^-8 each of what it rounds); scores (sums of 256 products in fp32) and exp2 add 1e-4 at most.
BOUND = 2.0 ** -7 * 1.05


def portions(layer, qkv, cuts):
    out, at = [], 0
    for n in cuts:
        out.append(layer.run(qkv[at:at + n], at)[0])
        at += n
    return np.concatenate(out)


@pytest.mark.parametrize("slope", [0.0, 0.02])
@pytest.mark.parametrize("heads,kv,dim,vdim,window,cuts", SHAPES)
def test_against_64_bits(heads, kv, dim, vdim, window, cuts, slope):
    total = sum(cuts)
    layer = Layer(heads, kv, dim, vdim, window, window + max(cuts) if window else total, slope=slope, seed=dim + window)          # a ring that wraps, where there is a window
    qkv, at = layer.inputs(total), 0
    for n in cuts:
        got, q = layer.run(qkv[at:at + n], at)
        want, size = layer.exact(q, at)
        assert (np.abs(got - want) <= BOUND * size + 1e-30).all(), (np.abs(got - want) / size).max()
        at += n


@pytest.mark.parametrize("heads,kv,dim,vdim,window,cuts", SHAPES)
def test_every_key_once(heads, kv, dim, vdim, window, cuts):
    """Value columns that add up the weights of every vdim-th position, near-uniform weights: a key that is missing, there twice or in sight of a row that must not
    see it changes a column by a tenth or more (some twenty positions a column at most)."""
    total = sum(cuts)
    layer = Layer(heads, kv, dim, vdim, window, window + max(cuts) if window else total, scale=0.1, seed=heads)
    qkv, at = layer.inputs(total), 0
    layer.values(qkv)[:] = (np.arange(total)[:, None] % vdim == np.arange(vdim)[None])[:, None, :]
    for n in cuts:
        got, q = layer.run(qkv[at:at + n], at)
        want, size = layer.exact(q, at)
        assert (np.abs(got - want) <= BOUND * size).all()
        at += n


@pytest.mark.parametrize("heads,kv,dim,vdim,cuts", [(4, 2, 64, 64, [2, 9, 140, 250]), (4, 2, 64, 64, [32, 369]), (8, 2, 128, 128, [255, 2, 600, 143]), (8, 2, 128, 128, [2, 18, 12, 33, 300]), (2, 2, 192, 130, [31, 2, 90]), (3, 1, 96, 80, [129, 42, 130]), (1, 1, 256, 256, [16, 17, 300, 65])])
def test_bits_under_any_cut(heads, kv, dim, vdim, cuts):
    """Without a window the tiles of keys begin at position 0, whatever the batch: a row's bits depend on its keys alone."""
    total = sum(cuts)
    whole, parts = (Layer(heads, kv, dim, vdim, 0, total, slope=0.01, scale=4.0, seed=3) for _ in "ab")
    qkv = whole.inputs(total)
    assert np.array_equal(whole.run(qkv, 0)[0], portions(parts, qkv, cuts))


@pytest.mark.parametrize("heads,kv,dim,vdim,window,cuts", SHAPES)
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_reach_of_a_value_that_is_not_finite(heads, kv, dim, vdim, window, cuts, bad):
    """Such a value stands in its column of the rows that see its key, and nowhere else: all other outputs keep their bits."""
    total = sum(cuts)
    make = lambda: Layer(heads, kv, dim, vdim, window, window + max(cuts) if window else total, slope=0.01, seed=7)  # noqa: E731
    clean = make()
    qkv = clean.inputs(total)
    spots = [(p, g, c) for p, g, c in ((0, 0, 0), (total // 3, kv - 1, vdim - 1), (total // 2, 0, vdim // 2), (total // 2 + 1, 0, vdim // 2 - 1), (total - 2, 0, 3))]
    want = portions(clean, qkv, cuts)
    marked = qkv.copy()
    for p, g, c in spots:
        clean.values(marked)[p, g, c] = bad
    got = portions(make(), marked, cuts)
    hit = np.zeros((total, heads, vdim), bool)
    for p, g, c in spots:
        last = total if window == 0 else min(total, p + window)
        hit[p:last, g * (heads // kv):(g + 1) * (heads // kv), c] = True
    assert np.array_equal(got[~hit], want[~hit])
    assert not np.isfinite(got[hit]).any()
    if not np.isnan(bad):
        assert (got[hit] == bad).all()
