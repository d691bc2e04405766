"""Kernels that are launched while their predecessor drains (llnv_set_pdl(1), the default) give what plain launches give, bit for
bit: buffers rewritten in every pass by kernels, copies and fills, work on two streams, calls from two threads."""
import threading

import pytest
import torch

import longlive_b200 as L
from longlive_b200 import _lib, dit, ops

pytestmark = pytest.mark.gpu


@pytest.fixture
def pdl():
    lib = _lib.lib()
    before = lib.llnv_set_pdl(1)
    yield lib.llnv_set_pdl
    lib.llnv_set_pdl(before)


def _bits(t):
    return t.clone().view(torch.uint8)


class Chain:
    """Quantize -> GEMM -> normalise and rotate -> cache write -> attention (window of two blocks and the chunk, split keys and their
    merge) -> dequantize, every buffer reused from pass to pass."""

    def __init__(self, seed, tokens=160, heads=2):
        g = torch.Generator(device="cuda").manual_seed(seed)
        c = heads * 128
        bf = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
        self.tokens, self.heads, self.c = tokens, heads, c
        self.inputs = [bf(tokens, c) * 2.0 ** (i % 5) for i in range(6)]
        self.w = ops.quantize_nvfp4(bf(3 * c, c), 3)
        self.bias, self.norm = bf(3 * c), bf(c)
        ang = torch.rand(tokens, 64, generator=g, device="cuda") * 6
        self.cos, self.sin = ang.cos().contiguous(), ang.sin().contiguous()
        self.x, self.qkv = torch.empty_like(self.inputs[0]), torch.empty(tokens, 3 * c, dtype=torch.bfloat16, device="cuda")
        self.blocks = [[L.quantize_to_fp4(bf(tokens * heads, 128)) for _ in range(2)] for _ in "kv"]
        self.q, self.k, self.out = (torch.empty_like(self.x) for _ in range(3))
        self.ws = torch.empty(ops.attention_nvfp4kv_workspace_bytes(tokens, 2, tokens, tokens, heads, key_splits=2), dtype=torch.uint8, device="cuda")
        self.amax = torch.empty(1, device="cuda")

    def step(self, i, keep):
        t, h, c = self.tokens, self.heads, self.c
        self.x.copy_(self.inputs[i % len(self.inputs)])
        codes, sf, amax = ops.quantize_nvfp4(self.x, 3)
        ops.gemm_nvfp4(codes, sf, amax, 3, *self.w, 3, t, 3 * c, c, out=self.qkv, bias=self.bias)
        q, k, v = (self.qkv[:, j * c:(j + 1) * c] for j in range(3))
        ops.rmsnorm_rope(q, self.norm, self.cos, self.sin, out=self.q)
        ops.rmsnorm_rope(k, self.norm, self.cos, self.sin, out=self.k)
        kv, vv = (s.reshape(t * h, 128) for s in (self.k, v))
        slot = i % 2
        for dst, src in zip(self.blocks, (kv, vv)):
            L.quantize_to_fp4(src, out=dst[slot])
        self.out.zero_()
        ops.attention_nvfp4kv(self.q, *self.blocks, t, self.k, v, h, out=self.out, key_splits=2, out_amax=self.amax, workspace=self.ws)
        y = ops.attention_bf16(self.out, self.k, v, h, key_splits=2)
        qo = ops.quantize_nvfp4(y, 3, self.amax)
        deq = ops.kv_dequant([b.values for b in self.blocks[0]], [b.scale_factors for b in self.blocks[0]], [b.amax for b in self.blocks[0]],
                             h, t, torch.bfloat16, 6, 256)
        if keep is not None:
            keep.append([_bits(x) for x in (self.out, y, qo[0], qo[1], self.amax, deq)])


def _same(a, b):
    assert len(a) == len(b)
    for x, y in zip(a, b):
        assert all(torch.equal(u, w) for u, w in zip(x, y))


def test_overlapped_launches_equal_plain_ones(pdl):
    runs = []
    for on in (0, 1, 1):
        pdl(on)
        chain, keep = Chain(1), []
        for i in range(40):
            chain.step(i, keep)
        torch.cuda.synchronize()
        runs.append(keep)
    _same(runs[0], runs[1])
    _same(runs[0], runs[2])


def test_overlapped_launches_on_two_streams(pdl):
    """Two chains on streams of their own, and a hand-over of one's output to the other through an event."""
    runs = []
    for on in (0, 1):
        pdl(on)
        a, b, keep_a, keep_b = Chain(1), Chain(2, tokens=300), [], []
        torch.cuda.synchronize()
        sa, sb = torch.cuda.Stream(), torch.cuda.Stream()
        for i in range(20):
            with torch.cuda.stream(sa):
                a.step(i, keep_a)
                done = sa.record_event()
            with torch.cuda.stream(sb):
                b.step(i, keep_b)
                sb.wait_event(done)
                keep_b.append([_bits(ops.quantize_nvfp4(a.out, 3)[0])])
                read = sb.record_event()
            sa.wait_event(read)
        torch.cuda.synchronize()
        runs.append((keep_a, keep_b))
    _same(runs[0][0], runs[1][0])
    _same(runs[0][1], runs[1][1])


def test_overlapped_launches_eager_model(pdl):
    cfg = dit.DiTConfig(dim=256, ffn_dim=512, heads=2, layers=3, text_len=128, text_dim=64, freq_dim=32, grid_h=6, grid_w=8,
                        frames_per_chunk=3, window_frames=9, sink_frames=3, in_channels=4)
    outs = []
    for on in (0, 1):
        pdl(on)
        model = dit.CausalDiT(cfg, seed=3)
        g = torch.Generator(device="cuda").manual_seed(4)
        ctx = model.encode_text(torch.randn(cfg.text_len, cfg.text_dim, generator=g, device="cuda").bfloat16())
        keep = []
        for chunk in range(4):
            x = torch.randn(cfg.chunk_tokens, cfg.patch_dim, generator=g, device="cuda").bfloat16()
            model.cache.begin_chunk()
            for t in (900.0, 500.0, 0.0):
                x = model.forward(x, torch.full((3,), t, device="cuda"), ctx, 3 * chunk, t_key=(t,) * 3).clone()
                keep.append([x.view(torch.uint8)])
        torch.cuda.synchronize()
        outs.append(keep)
    _same(outs[0], outs[1])


def test_calls_from_two_threads(pdl):
    want = []
    for seed in (1, 2):
        chain, keep = Chain(seed), []
        for i in range(20):
            chain.step(i, keep)
        want.append(keep)
    torch.cuda.synchronize()
    got, errors = [[], []], []

    def work(j):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                chain = Chain(1 + j)
                for i in range(20):
                    chain.step(i, got[j])
                torch.cuda.current_stream().synchronize()
        except Exception as exc:                          # noqa: BLE001 - reported by the test's own thread
            errors.append(exc)

    threads = [threading.Thread(target=work, args=(j,)) for j in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors
    _same(want[0], got[0])
    _same(want[1], got[1])


@pytest.mark.parametrize("op", ["quantize", "window"])
def test_a_blocked_launch_leaves_other_threads_running(op):
    """Behind half a second of device work the launch queue fills up and a launch blocks: meanwhile another Python thread goes on."""
    import time
    chain = Chain(1)
    codes, sf, amax = ops.quantize_nvfp4(chain.x, 3)
    if op == "quantize":
        call = lambda: ops.quantize_nvfp4(chain.x, 3, amax, codes, sf)
    else:
        call = lambda: ops.attention_nvfp4kv(chain.x, *chain.blocks, chain.tokens, chain.x, chain.x, chain.heads, out=chain.out, key_splits=2,
                                             workspace=chain.ws)
    call()
    torch.cuda.synchronize()
    stop, gaps = threading.Event(), []

    def tick():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.002)
            now = time.perf_counter()
            gaps.append(now - last)
            last = now

    ticker = threading.Thread(target=tick)
    ticker.start()
    torch.cuda._sleep(1_000_000_000)
    longest = 0.0
    for _ in range(3000):
        t0 = time.perf_counter()
        call()
        longest = max(longest, time.perf_counter() - t0)
    torch.cuda.synchronize()
    stop.set()
    ticker.join()
    assert longest > 0.1, "the launch queue never filled"
    assert max(gaps) < longest / 2


@pytest.mark.parametrize("m", [100, 1000, 4000])
def test_fp16_quantizer_overlapped_or_not(pdl, m):
    """The fp16 quantizer, whose launch overlaps its predecessor below and above a device full of CTAs but not between, reads what that
    predecessor wrote."""
    g = torch.Generator(device="cuda").manual_seed(m)
    w, xs = torch.eye(256, dtype=torch.bfloat16, device="cuda").repeat(12, 1), torch.randn(3, m, 256, generator=g, device="cuda").bfloat16()
    runs = []
    for on in (0, 1):
        pdl(on)
        x, keep = torch.empty(m, 3072, dtype=torch.float16, device="cuda"), []
        for i in range(6):
            x.copy_(ops.linear_bf16(xs[i % 3], w))
            ops.quantize_nvfp4(xs[(i + 1) % 3], 3)
            keep.append([_bits(t) for t in ops.quantize_nvfp4(x, 3)])
        torch.cuda.synchronize()
        runs.append(keep)
    _same(*runs)
