"""Kernels that a step takes by its size, each against the kernel it stands in for (the same bits, where it keeps every sum)
or against a float64 statement, at the sizes where it can go wrong: edges of tiles and chunks, remainders, one row and the most."""
import math
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def ops():
    from supersonic_b200.csrc import ops as o
    return o


def rnd(*shape, seed=0, scale=1.0, dtype=torch.float32):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (scale * torch.randn(*shape, device=DEV, generator=g)).to(dtype)


def off_by_one(t):
    """The same values at an address that no 16-byte access can take: the general kernel's operands."""
    flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    view = flat[1:].view(t.shape)
    view.copy_(t)
    return view


# rows that every form takes (one to sixteen rows a group, tiles), around the edges of groups, tiles, turns of 512 and chunks of 16
@pytest.mark.parametrize("m,n,k", [(1, 1, 4), (1, 9, 2052), (2, 130, 516), (3, 65, 20), (4, 8, 512), (5, 33, 1000), (8, 16, 528),
                                   (9, 200, 2048), (16, 64, 1028), (17, 100, 520), (33, 257, 300), (65, 130, 36), (129, 127, 44),
                                   (300, 2500, 516), (257, 129, 64), (64, 3, 4), (1000, 129, 12), (1000, 16400, 36),
                                   (1, 30001, 32), (1, 2500, 1028), (8, 2500, 516), (3, 9000, 1028), (7, 33000, 36), (16, 2500, 1028), (13, 8200, 516), (2, 5000, 2052),
                                   (2, 2500, 1028), (4, 2501, 516), (4, 9001, 2052), (4, 130, 8192), (2, 70, 9220), (1, 4000, 4),
                                   (2000, 9001, 260), (901, 2050, 2052), (700, 8200, 48), (520, 5000, 4)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_float32_products_are_the_general_kernels_bit_for_bit(m, n, k, accumulate):
    a, w, c = rnd(m, k, seed=m), rnd(n, k, seed=n), rnd(m, n, seed=k)
    a[0, k // 2] = 3e38                                             # a sum that overflows spreads the same way
    want, got = c.clone(), c.clone()
    ops().gemm_nt_plain(off_by_one(a), w, want, accumulate)
    ops().gemm_nt_plain(a, w, got, accumulate)
    assert torch.equal(torch.nan_to_num(got, nan=7.0), torch.nan_to_num(want, nan=7.0))
    wide = torch.full((m, n + 3), 5.0, device=DEV)                  # rows wider than the result: nothing beside it is touched
    ops().gemm_nt_plain(a, w, wide[:, :n], False)
    assert bool((wide[:, n:] == 5.0).all())


# tiles of 64 x 16 and of 32 x 32 whose chunks of k are shared out over warps: edges of tiles, turns of 8 chunks and chunks, blocks
# that walk several tiles
@pytest.mark.parametrize("m,n,k", [(64, 2100, 2052), (65, 2047, 20), (100, 1030, 516), (200, 2048, 1028), (17, 4700, 132), (32, 4700, 1028),
                                   (31, 9001, 148), (64, 3072, 128), (20, 16390, 264)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_float32_products_by_chunks_are_the_general_kernels_bit_for_bit(m, n, k, accumulate):
    test_float32_products_are_the_general_kernels_bit_for_bit(m, n, k, accumulate)


# more than 16 rows whose groups of 16 stay for several waves: partial groups, a last tile that is not full
@pytest.mark.parametrize("m,n,k", [(17, 3071, 2048), (32, 6144, 1024), (33, 5120, 8192), (80, 2558, 1024), (300, 512, 2544)])
def test_float32_products_of_groups_that_stay_are_the_general_kernels_bit_for_bit(m, n, k):
    test_float32_products_are_the_general_kernels_bit_for_bit(m, n, k, True)


@pytest.mark.parametrize("T,H,K,N", [(1, 6, 64, 128), (133, 3, 128, 48), (70, 4, 24, 72), (8, 2, 16, 260), (1000, 2, 68, 5000)])
def test_float32_head_products_are_the_general_kernels_bit_for_bit(T, H, K, N):
    x, w = rnd(T, H, K + 4, seed=T)[:, :, :K], rnd(H, N, K, seed=N)
    want, got = torch.empty(T, H, N, device=DEV), torch.empty(T, H, N, device=DEV)
    ops().head_linear_plain(off_by_one(x.contiguous()), w, want)
    ops().head_linear_plain(x, w, got)
    assert torch.equal(got, want)


@pytest.mark.parametrize("hd,v_dim,window,with_sinks", [(64, 64, 0, False), (128, 128, 0, True), (32, 32, 200, False), (20, 12, 0, False),
                                                        (128, 64, 129, True), (4, 4, 1, False)])
def test_float32_attention_with_staged_keys_is_the_plain_kernels_bit_for_bit(hd, v_dim, window, with_sinks):
    """Around whole chunks of 128 keys, rows of no slot, windows that start anywhere, values narrower than keys; pages that
    belong to nobody are not numbers, and one row sees an infinite value."""
    n_q, n_kv, pos, slots = 6, 2, [0, 126, 127, 128, 255, 256, 300, 5], [3, 0, 1, 2, 5, 4, 6, -1]
    perm = torch.randperm(40, generator=torch.Generator().manual_seed(hd)).to(torch.int32)
    table, at = torch.zeros(7, 6, dtype=torch.int32), 0
    k, v = rnd(40, n_kv, 64, hd, seed=1), rnd(40, n_kv, 64, v_dim, seed=2)
    for slot, p in zip(slots[:-1], pos):
        table[slot, :p // 64 + 1] = perm[at:at + p // 64 + 1]
        at += p // 64 + 1
    v[int(table[1, 1]), 0, 63, 1] = math.inf
    k[perm[at:].long()] = math.nan
    v[perm[at:].long()] = math.nan
    q = rnd(len(pos), n_q * hd, seed=3, scale=2.0)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    sinks = rnd(n_q, seed=4) if with_sinks else None
    outs = []
    for kc, vc in ((off_by_one(k), off_by_one(v)), (k, v)):
        out = torch.full((len(pos), n_q * v_dim), 9.0, device=DEV)
        ops().attention_plain(q, kc, vc, i32(pos), i32(slots), table.to(DEV), out, n_q, n_kv, hd, 6, window or None, hd ** -0.5,
                              value_dim=v_dim, sinks=sinks)
        outs.append(torch.nan_to_num(out, nan=7.0))
    assert torch.equal(outs[0], outs[1]) and bool((outs[1][-1] == 0).all())


@pytest.mark.parametrize("hd,rot,window", [(64, 64, 0), (128, 64, 0), (32, 32, 130), (20, 12, 0), (4, 0, 3), (128, 128, 128)])
def test_float32_decode_attention_rotates_and_appends_the_same_bits(hd, rot, window):
    """Against the two launches it stands in for: tokens at the edges of chunks and pages, one beyond the tables, one of no slot."""
    n_q, n_kv, pos, slots = 6, 2, [0, 63, 64, 127, 128, 300, 5], [3, 0, 1, 2, 5, 4, -1]
    table = torch.randperm(48, generator=torch.Generator().manual_seed(hd)).to(torch.int32)[:42].view(7, 6).to(DEV)
    k, v = rnd(48, n_kv, 64, hd, seed=1), rnd(48, n_kv, 64, hd, seed=2)
    cos, sin = rnd(290, rot // 2, seed=5), rnd(290, rot // 2, seed=6)
    qkv = rnd(len(pos), (n_q + 2 * n_kv) * hd + 3, seed=3, scale=2.0)[:, : (n_q + 2 * n_kv) * hd]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    p, s, o = i32(pos), i32(slots), ops()
    want_k, want_v, want_q, want = k.clone(), v.clone(), qkv.clone(), torch.empty(len(pos), n_q * hd, device=DEV)
    o.rope_append(want_q, cos if rot else None, sin if rot else None, p, s, table, want_k, want_v, n_q, n_kv, hd, rot, 6)
    o.attention_plain(want_q, want_k, want_v, p, s, table, want, n_q, n_kv, hd, 6, window or None, hd ** -0.5)
    got, before = torch.full_like(want, 9.0), qkv.clone()
    o.attention_f32_decode(qkv, cos, sin, k, v, p, s, table, got, n_q, n_kv, hd, rot, 6, window or None, hd ** -0.5)
    assert torch.equal(got, want) and torch.equal(k, want_k) and torch.equal(v, want_v) and torch.equal(qkv, before)


# blocks (a token and a head each) for two, three, four and more a multiprocessor: rings of every depth, slices and stages that are
# not full, heads that keep whole chunks while they fit
@pytest.mark.parametrize("blocks", [2, 3, 4, 7])
@pytest.mark.parametrize("hd,v_dim,window,with_sinks", [(64, 64, 0, False), (128, 128, 0, True), (128, 64, 129, False), (96, 96, 0, False), (64, 100, 1, True),
                                                        (36, 20, 200, False)])
def test_float32_attention_of_many_rows_is_the_plain_kernels_bit_for_bit(blocks, hd, v_dim, window, with_sinks):
    o, n_q, n_kv, slots = ops(), 6, 2, 7
    T = o.sm_count() * blocks // n_q - 3
    pages = 6
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    pos, slot = i32([(t * 37 + 126) % 380 for t in range(T)]), i32([-1 if t % 40 == 11 else t % slots for t in range(T)])
    table = torch.randperm(slots * pages, generator=torch.Generator().manual_seed(hd)).to(torch.int32).view(slots, pages).to(DEV)
    k, v = rnd(slots * pages, n_kv, 64, hd, seed=1), rnd(slots * pages, n_kv, 64, v_dim, seed=2)
    v[int(table[1, 5]), 0, 63, 1] = math.inf
    q, sinks = rnd(T, n_q * hd, seed=3, scale=2.0), rnd(n_q, seed=4) if with_sinks else None
    outs = []
    for kc, vc in ((off_by_one(k), off_by_one(v)), (k, v)):
        out = torch.full((T, n_q * v_dim), 9.0, device=DEV)
        o.attention_plain(q, kc, vc, pos, slot, table, out, n_q, n_kv, hd, 6, window or None, hd ** -0.5, value_dim=v_dim, sinks=sinks)
        outs.append(torch.nan_to_num(out, nan=7.0))
    assert torch.equal(*outs)


@pytest.mark.parametrize("blocks", [2, 3, 4, 7])
@pytest.mark.parametrize("hd,rot,window", [(64, 64, 0), (128, 64, 0), (96, 12, 130), (36, 0, 3)])
def test_float32_decode_attention_of_many_sequences_rotates_and_appends_the_same_bits(blocks, hd, rot, window):
    """Against the two launches it stands in for, around whole chunks and pages, with rows of no slot."""
    o, n_q, n_kv = ops(), 6, 2
    T = o.sm_count() * blocks // n_q - 3
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    edges = [0, 31, 32, 63, 64, 127, 128, 159, 255, 256, 300, 319]
    pos, slot = i32([edges[t % len(edges)] for t in range(T)]), i32([-1 if t % 40 == 11 else t for t in range(T)])
    table = torch.randperm(5 * T, generator=torch.Generator().manual_seed(hd)).to(torch.int32).view(T, 5).to(DEV)
    k, v = rnd(5 * T, n_kv, 64, hd, seed=1), rnd(5 * T, n_kv, 64, hd, seed=2)
    cos, sin = rnd(310, rot // 2, seed=5), rnd(310, rot // 2, seed=6)
    qkv = rnd(T, (n_q + 2 * n_kv) * hd, seed=3, scale=2.0)
    want_k, want_v, want_q, want = k.clone(), v.clone(), qkv.clone(), torch.empty(T, n_q * hd, device=DEV)
    o.rope_append(want_q, cos if rot else None, sin if rot else None, pos, slot, table, want_k, want_v, n_q, n_kv, hd, rot, 6)
    o.attention_plain(want_q, off_by_one(want_k), off_by_one(want_v), pos, slot, table, want, n_q, n_kv, hd, 6, window or None, hd ** -0.5)
    got, before = torch.full_like(want, 9.0), qkv.clone()
    o.attention_f32_decode(qkv, cos, sin, k, v, pos, slot, table, got, n_q, n_kv, hd, rot, 6, window or None, hd ** -0.5)
    assert torch.equal(got, want) and torch.equal(k, want_k) and torch.equal(v, want_v) and torch.equal(qkv, before)


@pytest.mark.parametrize("m,inter,k", [(1, 5, 2052), (2, 2001, 520), (3, 901, 36), (4, 1000, 1028), (2, 8192, 2048), (1, 1801, 64)])
@pytest.mark.parametrize("kind,limit", [("silu", 0.0), ("clamped_swish", 2.0), ("gelu_tanh", 0.0)])
def test_float32_gated_products_are_the_two_launches_bit_for_bit(m, inter, k, kind, limit):
    x, w, scale = rnd(m, k, seed=m), rnd(2 * inter, k, seed=inter, scale=0.1), rnd(m, seed=k)
    if not ops().gemm_f32_gated_ok(x, w, torch.empty(m, inter, device=DEV)):
        pytest.skip("another kernel makes this product")
    both, want, got = torch.empty(m, 2 * inter, device=DEV), torch.empty(m, inter, device=DEV), torch.empty(m, inter, device=DEV)
    for factor in (None, scale):
        ops().gemm_nt_plain(x, w, both)
        ops().gated_activation(both, want, kind, limit, row_scale=factor)
        ops().gemm_f32_gated(x, w, got, kind, limit, factor)
        assert torch.equal(got, want)


@pytest.mark.parametrize("hd,n_q,n_kv", [(64, 8, 2), (128, 6, 2), (128, 3, 3), (64, 12, 1)])
def test_float32_prompt_attention_is_the_plain_kernels_bit_for_bit(hd, n_q, n_kv):
    """Prompts that continue a cache, of one token, of exactly a chunk of keys and a page; pages that belong to nobody are
    not numbers, and the last value of a sequence is infinite: only the rows that see it may be."""
    lens, starts, slots = [100, 300, 1, 128, 9, 64], [0, 64, 200, 0, 119, 128], [4, 0, 2, 5, 1, 3]
    T, pages = sum(lens), sum((n + s + 63) // 64 for n, s in zip(lens, starts))
    perm = torch.randperm(pages + 3, generator=torch.Generator().manual_seed(hd)).to(torch.int32)
    table, at = torch.zeros(6, 16, dtype=torch.int32), 0
    k, v = rnd(pages + 3, n_kv, 64, hd, seed=1), rnd(pages + 3, n_kv, 64, hd, seed=2)
    for slot, n, s in zip(slots, lens, starts):
        need = (n + s + 63) // 64
        table[slot, :need] = perm[at:at + need]
        at += need
        v[int(table[slot, need - 1]), 0, (n + s - 1) % 64, 3] = math.inf
    k[perm[at:].long()] = math.nan
    v[perm[at:].long()] = math.nan
    q = rnd(T, n_q * hd + 64, seed=3, scale=2.0)[:, : n_q * hd]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    pos = torch.cat([torch.arange(s, s + n) for n, s in zip(lens, starts)]).to(torch.int32).to(DEV)
    slot_of = torch.cat([torch.full((n,), s) for n, s in zip(lens, slots)]).to(torch.int32).to(DEV)
    cu = i32([sum(lens[:i]) for i in range(len(lens) + 1)])
    want, got = torch.empty(T, n_q * hd, device=DEV), torch.full((T, n_q * hd), 7.0, device=DEV)
    assert ops().attention_f32_prompt_ok(q, k, v, got, hd)
    ops().attention_plain(q, k, v, pos, slot_of, table.to(DEV), want, n_q, n_kv, hd, 6, None, hd ** -0.5)
    ops().attention_f32_prompt(q, k, v, cu, i32(starts), i32(slots), table.to(DEV), got, max(lens), n_q, n_kv, hd, 6, hd ** -0.5)
    assert bool(torch.isinf(want).any())
    assert torch.equal(torch.nan_to_num(got, nan=7.0), torch.nan_to_num(want, nan=7.0))


@pytest.mark.parametrize("H,dk,dv,window", [(16, 576, 512, None), (16, 576, 512, 100), (8, 288, 256, None), (6, 224, 192, 96),
                                            (3, 400, 384, 7), (5, 48, 32, None), (1, 64, 16, 64)])
def test_latent_attention_of_prompts_on_tcgen05(H, dk, dv, window):
    """Against float64 attention over the same bfloat16 rows: as close as the mma.sync kernel (both round their result to
    bfloat16 and keep 16 bits of a weight, so the error is the result's rounding: 2^-9 relative, root mean square)."""
    from test_sotavik_kernels_gpu import latent_case, latent_reference
    o, scale = ops(), dk ** -0.5
    for lengths, new, sinks in (([200, 65, 1, 130], [70, 65, 1, 3], None), ([300, 64, 129], [300, 1, 129], torch.linspace(-1.0, 2.0, H, device=DEV))):
        cache, batch, store, table, q, rows = latent_case(lengths, new, H, dk, dv, seed=H + dk)
        T = sum(new)
        ref = latent_reference(q, rows, lengths, new, H, dk, dv, scale, sinks, window).double()
        out = torch.full((T, H * dv), 7.0, dtype=torch.bfloat16, device=DEV)
        assert o.latent_attention_tc_ok(q, store, out, H, dk, dv, 6)
        o.latent_attention_tc(q, store, batch.cu_new, batch.seq_start, batch.seq_slot, table, out, sinks, batch.max_new, H, dk, dv,
                              6, window, scale)
        torch.cuda.synchronize()
        o.check_device_errors(torch.device(DEV))
        err = float((out.double() - ref).norm() / ref.norm())
        assert err < 2.0 ** -9, (lengths, new, err)


@pytest.mark.parametrize("H,dk,dv,window", [(16, 576, 512, None), (8, 288, 256, None), (5, 48, 32, None), (16, 576, 512, 150), (3, 96, 64, 100)])
@pytest.mark.parametrize("sinked", [False, True])
def test_latent_attention_moves_its_reference_with_scores_that_grow(H, dk, dv, window, sinked):
    """Keys that grow along the sequence, at another pace for every head and token: a row's weights outgrow the maximum of its
    first keys in several turns, in some rows of a warp and not in others, and what was summed against the old maximum is
    scaled by a factor between zero and one.  Row by row against float64: the result's rounding to bfloat16, 2^-9 of every
    element, and weights of 16 bits."""
    from test_sotavik_kernels_gpu import latent_case
    o, scale, lengths, new = ops(), dk ** -0.5, [420, 200, 64, 333], [300, 170, 64, 1]
    cache, batch, store, table, q, rows = latent_case(lengths, new, H, dk, dv, seed=H + dk)
    sinks = torch.linspace(-1.0, 6.0, H, device=DEV) if sinked else None
    lean = rnd(dk, seed=3)
    T = sum(new)
    with_lean = torch.rand(T, H, 1, device=DEV, generator=torch.Generator(device=DEV).manual_seed(4)) * 3.0
    q.copy_((q.view(T, H, dk).float() * 0.5 + with_lean * lean * dk ** -0.5 * 4.0).to(torch.bfloat16).view(T, H * dk))
    moved, stayed, at = 0, 0, 0
    out = torch.full((T, H * dv), math.nan, dtype=torch.bfloat16, device=DEV)
    want = torch.empty(T, H, dv, dtype=torch.float64, device=DEV)
    for b, (n, k) in enumerate(zip(lengths, new)):
        p = torch.arange(n, device=DEV)
        r = (rows[b].float() * 0.5 + (p[:, None] / 64.0).floor() * 0.5 * lean).to(torch.bfloat16)
        slot = int(batch.seq_slot[b])
        for page in range((n + 63) // 64):
            piece = r[64 * page:64 * page + 64]
            store[int(table[slot, page]), 0, : piece.shape[0]] = piece
        s = torch.einsum("thd,kd->thk", q[at:at + k].double().view(k, H, dk), r.double()) * scale
        pos = torch.arange(n - k, n, device=DEV)[:, None]
        seen = (p[None] <= pos) & ((p[None] > pos - window) if window else (p[None] >= 0))
        s = s.masked_fill(~seen[:, None], -math.inf)
        w = torch.exp(s - s.amax(2, keepdim=True))
        den = w.sum(2) + (torch.exp(sinks.double()[None] - s.amax(2)) if sinked else 0.0)
        want[at:at + k] = torch.einsum("thk,kv->thv", w, r[:, :dv].double()) / den[:, :, None]
        if n > 128:                                    # pages of the last tokens against the maximum of their first one
            pages = torch.nn.functional.pad(s[-60:], (0, -n % 64), value=-math.inf).view(min(k, 60), H, -1, 64)
            first = pages.amax(3).gather(2, torch.isfinite(pages.amax(3)).int().argmax(2, keepdim=True))
            grown = (torch.exp(pages - first[..., None]).sum(3) > 256.0).any(2)
            moved, stayed = moved + int(grown.sum()), stayed + int((~grown).sum())
        at += k
    assert moved > 20 and stayed > 20, (moved, stayed)
    o.latent_attention_tc(q, store, batch.cu_new, batch.seq_start, batch.seq_slot, table, out, sinks, batch.max_new, H, dk, dv, 6,
                          window, scale)
    o.check_device_errors(torch.device(DEV))
    err = (out.double().view(T, H, dv) - want).norm(dim=2) / want.norm(dim=2)
    assert float(err.max()) < 2.0 ** -8, float(err.max())


def test_latent_attention_of_prompts_ends_with_its_last_sums():
    """Prompts of one to six turns with the shortest products, where the last two weighted sums end close together: run many
    times, every row is written each time, with the same bits, and no wait runs out."""
    from test_sotavik_kernels_gpu import latent_case
    o, H, dk, dv = ops(), 16, 48, 32
    for lengths in ([8, 64, 65, 128, 129, 190], [192, 193, 256, 257, 320, 384]):
        cache, batch, store, table, q, rows = latent_case(lengths, lengths, H, dk, dv, seed=sum(lengths))
        first = None
        for turn in range(200):
            out = torch.full((sum(lengths), H * dv), math.nan, dtype=torch.bfloat16, device=DEV)
            o.latent_attention_tc(q, store, batch.cu_new, batch.seq_start, batch.seq_slot, table, out, None, batch.max_new, H, dk, dv,
                                  6, None, dk ** -0.5)
            first = out if first is None else first
            assert torch.equal(out, first), (lengths, turn)
        o.check_device_errors(torch.device(DEV))
        assert bool(torch.isfinite(first).all())


@pytest.mark.parametrize("rows,n,k", [(1, 16, 64), (1, 3072, 2048), (7, 200, 448), (16, 33, 64), (16, 4736, 576), (3, 8200, 1088), (2, 1000, 8192),
                                      (9, 12000, 192)])
@pytest.mark.parametrize("tile", [16, 32, 64])
def test_products_of_few_rows_in_narrow_tiles(rows, n, k, tile):
    """Tiles of W that are not whole, stages whose last k-blocks do not exist, rows beyond the step's that must stay as they are:
    float32 sums of bfloat16 products, 1e-5 of the result's norm, and one rounding where they are stored."""
    x, w = rnd(rows, k, seed=rows, dtype=torch.bfloat16), rnd(n, k, seed=n, scale=0.05, dtype=torch.bfloat16)
    x = torch.cat([x, torch.full((rows, 8), math.nan, dtype=torch.bfloat16, device=DEV)], dim=1)[:, :k]        # rows 16 bytes apart
    want = x.double() @ w.double().T
    o = ops()
    got = torch.full((rows + 1, n), 3.0, device=DEV)
    o.gemv_rows(x, w, got[:rows], tile)
    assert float((got[:rows] - want).norm() / want.norm()) < 1e-5 and bool((got[rows] == 3.0).all())
    got = torch.empty(rows, n + 8, dtype=torch.bfloat16, device=DEV)[:, :n]
    o.gemv_rows(x, w, got, tile, act="relu_squared", scale=0.5)
    ref = (0.5 * want.clamp(min=0) ** 2)
    assert float((got.double() - ref).norm() / ref.norm()) < 2.0 ** -8          # half a unit in the last of eight bits, at most
    o.check_device_errors(torch.device(DEV))


@pytest.mark.parametrize("hd,lens", [(64, [300] * 60 + [450] * 14), (64, [20, 330] * 40), (128, [700] * 30), (128, [64 * 40] * 5 + [3]),
                                     (64, [400] * 100), (128, [1, 64, 65, 320, 321, 384, 385])])
def test_decode_attention_cuts_its_sequences_itself(hd, lens):
    """One item a block where some size of chunk allows it, none does, five pages or fewer, a padding row: the outputs of the
    same keys in fixed chunks of three pages, within the rounding of the weights to bfloat16 (2^-8 of a value)."""
    o, n_q, n_kv, B = ops(), 8, 4, len(lens)
    pages = [(n + 63) // 64 for n in lens]
    most, at = max(pages), 0
    perm = torch.randperm(sum(pages), generator=torch.Generator().manual_seed(hd)).to(torch.int32)
    table = torch.zeros(B, most, dtype=torch.int32)
    for b, n in enumerate(pages):
        table[b, :n] = perm[at:at + n]
        at += n
    k, v = rnd(sum(pages), n_kv, 64, hd, seed=1, dtype=torch.bfloat16), rnd(sum(pages), n_kv, 64, hd, seed=2, dtype=torch.bfloat16)
    q = rnd(B, n_q * hd, seed=3, dtype=torch.bfloat16)
    slots = list(range(B))
    slots[1] = -1
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    outs = []
    for chunk in (3, 0):
        chunks = -(-most // 2)
        nf, nc = o.attention_decode_chunked_scratch(B, n_q, n_kv, hd, chunks)
        scratch, counters = torch.full((nf,), math.nan, device=DEV), torch.zeros(nc, dtype=torch.int32, device=DEV)
        out = torch.full((B, n_q * hd), 9.0, dtype=torch.bfloat16, device=DEV)
        o.attention_decode_chunked(q, k, v, i32([n - 1 for n in lens]), i32(slots), table.to(DEV), out, n_q, n_kv, hd, 6, None,
                                   hd ** -0.5, chunk, chunks, scratch, counters)
        assert bool((counters == 0).all())
        outs.append(out.float())
    assert bool((outs[1][1] == 0).all())
    assert float((outs[0] - outs[1]).norm() / outs[0].norm()) < 2.0 ** -8
    o.check_device_errors(torch.device(DEV))


@pytest.mark.parametrize("hd,n_q,n_kv", [(64, 32, 8), (128, 32, 8), (128, 24, 8)])
def test_decode_attention_cuts_a_long_sequence_beside_short_ones(hd, n_q, n_kv):
    """So many short sequences that only uncut items would be taken in one go: the long one's parts still meet through the
    scratch (uncut it keeps one block busy six times as long as the others take together)."""
    o = ops()
    B = o.sm_count() * 2 // n_kv - 5                                # of two blocks a multiprocessor, all but a few have an item
    lens = [100] * (B - 1) + [8000]
    k, v = (rnd(125, n_kv, 64, hd, seed=s, dtype=torch.bfloat16) for s in (1, 2))
    table = torch.arange(125, dtype=torch.int32, device=DEV).repeat(B, 1)
    q, out = rnd(B, n_q * hd, seed=3, dtype=torch.bfloat16), torch.empty(B, n_q * hd, dtype=torch.bfloat16, device=DEV)
    chunks = o.sm_count() * 2 // n_kv
    nf, nc = o.attention_decode_chunked_scratch(B, n_q, n_kv, hd, chunks)
    scratch, counters = torch.full((nf,), math.nan, device=DEV), torch.zeros(nc, dtype=torch.int32, device=DEV)
    o.attention_decode_chunked(q, k, v, torch.tensor([n - 1 for n in lens], dtype=torch.int32, device=DEV),
                               torch.arange(B, dtype=torch.int32, device=DEV), table, out, n_q, n_kv, hd, 6, None, hd ** -0.5, 0, chunks,
                               scratch, counters)
    o.check_device_errors(torch.device(DEV))
    assert bool((~scratch.isnan()).any())


@pytest.mark.parametrize("hd,n_q,n_kv,T", [(64, 8, 2, 37), (128, 6, 3, 5), (64, 32, 8, 131), (8, 1, 1, 1)])
def test_rotation_from_split_sums_is_the_two_launches_bit_for_bit(hd, n_q, n_kv, T):
    """Rounding, rotation and append in one pass; a padding row's sums are cleared and nothing else."""
    o, n = ops(), (n_q + 2 * n_kv) * hd
    sums0, cos, sin = rnd(T, n, seed=1, scale=3.0), rnd(T + 5, hd // 2, seed=2), rnd(T + 5, hd // 2, seed=3)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    pos, slot = i32(list(range(5, T + 5))), i32([0 if t != 3 else -1 for t in range(T)])
    table = torch.randperm(4, generator=torch.Generator().manual_seed(hd)).to(torch.int32).view(1, 4).to(DEV)
    caches = [[rnd(4, n_kv, 64, hd, seed=4, dtype=torch.bfloat16) for _ in range(2)] for _ in range(2)]
    sums, want, got = sums0.clone(), torch.empty(T, n, dtype=torch.bfloat16, device=DEV), torch.full((T, n), 7.0, dtype=torch.bfloat16, device=DEV)
    o.round_and_clear(sums, want)
    o.rope_append_vec(want, cos, sin, pos, slot, table, *caches[0], n_q, n_kv, hd, 6)
    sums = sums0.clone()
    o.rope_append_sums(sums, got, cos, sin, pos, slot, table, *caches[1], n_q, n_kv, hd, 6)
    live = (slot >= 0).cpu()
    assert torch.equal(got[:, :n_q * hd].cpu()[live], want[:, :n_q * hd].cpu()[live]) and bool((got[:, n_q * hd:] == 7.0).all())
    assert bool((sums == 0).all()) and all(torch.equal(a, b) for a, b in zip(*caches))


@pytest.mark.parametrize("top_k", [1, 5, 40, 64])
@pytest.mark.parametrize("top_p,vocab", [(1.0, 70001), (0.9, 70001), (0.6, 70001), (0.0, 70001), (0.9, 50), (1.0, 65), (0.6, 4096), (0.9, 400000)])
def test_a_row_draws_the_same_token_from_its_candidates_as_from_the_held_row(top_k, top_p, vocab):
    """A cut of a large step is searched over candidates, of a small one over the row: the same tokens.  Rows with ties at the
    cut, everything tied (more candidates than are kept: both cuts over the row, its weights made again in every pass), one
    huge token, few finite ones, not-a-numbers."""
    n = 18
    lg = rnd(n, vocab, seed=top_k, scale=2.5)
    lg[0] = (lg[0] * 2).round() / 2
    lg[1, :] = 1.25
    lg[2, vocab // 2] = 90.0
    lg[3, 30:] = -math.inf
    lg[4, 17] = math.nan
    lg[5] = lg[5].sort(descending=True).values
    lg[8] = 1.25 - (torch.arange(vocab, device=DEV) % 3 == 0).float()
    lg[6, :] = -math.inf
    lg[7, 9] = math.inf
    seeds = torch.arange(1, n + 1, dtype=torch.int64, device=DEV) * 0x1E3779B97F4A7C15
    drawn = []
    for form in (1, 2, 0):
        state, out, u = seeds.clone(), torch.empty(n, dtype=torch.int32, device=DEV), torch.empty(n, device=DEV)
        for turn in range(3):
            ops().sample(lg, 0.7, top_k, top_p, None, state, out, u, form=form)
            drawn.append(torch.cat([out, u.view(torch.int32)]))
    for turn in range(3):
        assert torch.equal(drawn[turn], drawn[3 + turn]) and torch.equal(drawn[turn], drawn[6 + turn])
    for lo in range(0, n, 9):
        alone, got = seeds[lo:lo + 9].clone(), torch.empty(9, dtype=torch.int32, device=DEV)
        ops().sample(lg[lo:lo + 9].contiguous(), 0.7, top_k, top_p, None, alone, got)
        assert torch.equal(got, drawn[0][lo:lo + 9])


@pytest.mark.parametrize("H,d,dv", [(4, 256, 512), (3, 40, 24), (2, 128, 72), (1, 200, 30), (2, 65, 33)])
def test_gated_scan_in_register_tiles(H, d, dv):
    """Runs long and short of whole turns of eight tokens, whole and in chunks, against the recurrence in float64; float32
    sums of d terms after hundreds of float32 state updates: 2e-6 relative."""
    lens = [70, 9, 133]
    T, B = sum(lens), len(lens)
    proj, z0, bias = rnd(T, 2 * H * d + H * dv, seed=d), rnd(T, H * d, seed=1), rnd(H * d, seed=2) + 1.0
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    cu, slots, state0 = i32([0, 70, 79, 212]), i32([2, 0, 3]), rnd(4, H * d * dv, seed=3)
    decay = (torch.sigmoid((z0 + bias).double()) ** (1 / 16)).view(T, H, d)
    q, k, v = proj[:, :H * d].double().view(T, H, d), proj[:, H * d:2 * H * d].double().view(T, H, d), proj[:, 2 * H * d:].double().view(T, H, dv)
    want, end, at = torch.empty(T, H, dv, dtype=torch.float64, device=DEV), state0.double().view(4, H, d, dv).clone(), 0
    for slot, n in zip((2, 0, 3), lens):
        S = end[slot]
        for t in range(at, at + n):
            S = decay[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :]
            want[t] = torch.einsum("hdv,hd->hv", S, q[t]) * 0.25
        end[slot] = S
        at += n
    for chunk, form in ((0, 0), (24, 0), (64, 0), (0, 1), (24, 1)) + (((0, 2), (24, 2), (64, 2)) if d > 64 else ()) + \
            (((0, 3),) if dv % 4 == 0 else ()):
        n = -(-max(lens) // chunk) if chunk else 0
        sums = torch.empty(max(B * n * H * d * dv, 1), device=DEV)
        decays = torch.empty(max(B * n * H * d, 1), device=DEV)
        state, z, out = state0.clone(), z0.clone(), torch.empty(T, H * dv, device=DEV)
        ops().gated_linear_scan(proj, 0, H * d, 2 * H * d, z, bias, 16.0, 0.25, state, cu, slots, out, H, d, dv, chunk=chunk,
                                max_new=max(lens), sums=sums if chunk else None, decays=decays if chunk else None, form=form)
        assert float((out.double() - want.view(T, -1)).norm() / want.norm()) < 2e-6, chunk
        assert float((state.double().view(-1) - end.view(-1)).norm() / end.norm()) < 2e-6, chunk


@pytest.mark.parametrize("B,H,d,dv", [(3, 2, 256, 512), (80, 4, 100, 132), (1, 3, 33, 4), (75, 1, 256, 260)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_gated_scan_of_one_token_a_sequence(B, H, d, dv, dtype):
    """A decode step by rows of the state, in narrow and in wide blocks, a padding row among them, against the walk."""
    proj, z0, bias = rnd(B, 2 * H * d + H * dv, seed=d, dtype=dtype), rnd(B, H * d, seed=1), rnd(H * d, seed=2) + 1.0
    cu = torch.arange(B + 1, dtype=torch.int32, device=DEV)
    slots = torch.randperm(B + 1, generator=torch.Generator().manual_seed(B)).to(torch.int32)[:B].to(DEV)
    if B > 1:
        slots[B // 2] = -1
    state0, got = rnd(B + 1, H * d * dv, seed=3), []
    for form in (1, 0):
        state, out = state0.clone(), torch.zeros(B, H * dv, device=DEV)
        ops().gated_linear_scan(proj, 0, H * d, 2 * H * d, z0.clone(), bias, 16.0, 0.25, state, cu, slots, out, H, d, dv, form=form)
        got.append((out, state))
    assert torch.equal(got[0][1], got[1][1])                       # a state's element is one product and one multiply-add
    assert float((got[0][0] - got[1][0]).norm() / got[0][0].norm()) < 1e-6       # sums of d float32 products in another order


@pytest.mark.parametrize("H,d,dv,lens", [(4, 100, 132, [5] * 80), (3, 128, 64, [1, 9, 30, 2] * 15), (1, 65, 260, [12] * 40)])
def test_gated_scan_is_the_same_bits_whatever_shares_a_multiprocessor(H, d, dv, lens):
    """So many sequences that two blocks share a multiprocessor, and each of them alone, in the form that does not go by the sizes."""
    o, width = ops(), 2 * H * d + H * dv
    T, at = sum(lens), [sum(lens[:i]) for i in range(len(lens) + 1)]
    proj, z, bias = rnd(T, width, seed=1, dtype=torch.bfloat16), rnd(T, H * d, seed=2), rnd(H * d, seed=3) + 1.0
    state0 = rnd(len(lens), H * d * dv, seed=4)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731

    def run(which):
        rows = slice(at[which[0]], at[which[-1] + 1])
        state, out = state0.clone(), torch.full((rows.stop - rows.start, H * dv), math.nan, device=DEV)
        o.gated_linear_scan(proj[rows], 0, H * d, 2 * H * d, z[rows].clone(), bias, 16.0, 0.25, state, i32([at[i] - rows.start for i in which] + [rows.stop - rows.start]),
                            i32(which), out, H, d, dv, form=1)
        return out, state
    together, end = run(list(range(len(lens))))
    for i in range(0, len(lens), 7):
        out, state = run([i])
        assert torch.equal(out, together[at[i]:at[i + 1]]) and torch.equal(state[i], end[i])


@pytest.mark.parametrize("H,d,dv,lens", [(4, 256, 512, [2]), (2, 100, 132, [2, 1, 2]), (1, 40, 24, [1, 2] * 40), (3, 65, 30, [2, 2])])
def test_gated_scan_of_two_tokens_a_sequence(H, d, dv, lens):
    """The serving set's choice for them against the recurrence in 64 bits: sums of d products in float32 (2^-24 each)."""
    from supersonic_b200.csrc.fast_sets import FastKernels
    T, batch = sum(lens), step_of(lens, list(range(len(lens)))[::-1])
    proj, z, bias = rnd(T, 2 * H * d + H * dv, seed=1, dtype=torch.bfloat16), rnd(T, H * d, seed=2), rnd(H * d, seed=3) + 1.0
    state, out = rnd(len(lens), H * d * dv, seed=4), torch.full((T, H * dv), math.nan, device=DEV)
    S, want, t = state.double().view(-1, H, d, dv).clone(), torch.empty(T, H, dv, dtype=torch.float64, device=DEV), 0
    q, k, v = (x.double() for x in (proj[:, :H * d].view(T, H, d), proj[:, H * d:2 * H * d].view(T, H, d), proj[:, 2 * H * d:].view(T, H, dv)))
    decay = torch.sigmoid(z.double() + bias.double()).pow(1 / 16.0).view(T, H, d)
    for i, n in enumerate(lens):
        s = len(lens) - 1 - i
        for t in range(t, t + n):
            S[s] = decay[t][..., None] * S[s] + k[t][..., None] * v[t][:, None]
            want[t] = torch.einsum("hd,hdv->hv", 0.25 * q[t], S[s])
        t += 1
    FastKernels().gated_linear_scan(proj, 0, H * d, 2 * H * d, z, bias, 16.0, 0.25, state, batch, out, H, d, dv)
    assert float((out.double() - want.view(T, -1)).norm() / want.norm()) < d ** 0.5 * 2.0 ** -23
    assert float((state.double() - S.view_as(state)).norm() / S.norm()) < 2.0 ** -21


def step_of(lens, slots):
    """What a kernel set reads of a step of new tokens, sequence ``i`` bringing ``lens[i]`` in ``slots[i]``."""
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    return SimpleNamespace(n_seqs=len(lens), n_tokens=sum(lens), max_new=max(lens), is_decode=max(lens) == 1, seq_slot=i32(slots),
                           cu_new=i32([sum(lens[:i]) for i in range(len(lens) + 1)]))


@pytest.mark.parametrize("form", ["gated", "tied", "tied wide"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_a_deterministic_sets_scan_depends_on_no_other_sequence(form, dtype, monkeypatch):
    """Sequences of fewer tokens than are cut, of just as many and of more, alone, beside one another, and with a scratch that
    holds fewer chunks than the step has: outputs and states are the same bits.  The serving set's own cut, which does depend
    on the step, stays within float32 rounding of them."""
    o, H, d, dv = ops(), 2, 64, 160 if form == "tied wide" else 64
    from supersonic_b200.csrc.fast_sets import FastKernels
    lens, slots = [200, 300, 1, 256, 255, 700, 60], [3, 0, 6, 1, 5, 2, 4]
    T, width = sum(lens), 2 * H * d + H * dv
    rows, z0, bias = rnd(T, width, seed=1, dtype=dtype), rnd(T, H * d, seed=2), rnd(H * d, seed=3) + 1.0
    state0, lower, gain = rnd(7, H * d * dv, seed=4), torch.rand(H * d, device=DEV) * 0.9, rnd(dv, seed=5)

    def run(which, deterministic=True):
        ks, at = FastKernels(deterministic=deterministic), [sum(lens[:i]) for i in which]
        take = torch.cat([torch.arange(a, a + lens[i]) for a, i in zip(at, which)]).to(DEV)
        batch, state, proj = step_of([lens[i] for i in which], [slots[i] for i in which]), state0.clone(), rows[take]
        if form == "gated":
            out = torch.full((len(take), H * dv), math.nan, device=DEV)
            ks.gated_linear_scan(proj, 0, H * d, 2 * H * d, z0[take], bias, 16.0, 0.25, state, batch, out, H, d, dv)
        else:
            out = torch.full((len(take), H * dv), math.nan, device=DEV, dtype=dtype)
            ks.tied_scan(proj, 0, H * d, 2 * H * d, bias, lower, state, batch, gain, 1e-5, out, H, d, dv)
        return list(out.split([lens[i] for i in which])), state
    together, end = run(range(len(lens)))
    for group in ([0], [1], [5], [0, 1], [4, 3, 6], [2, 5, 0], [6, 5]):
        outs, states = run(group)
        for i, out in zip(group, outs):
            assert torch.equal(out, together[i]) and torch.equal(states[slots[i]], end[slots[i]]), (group, i)
    for places in (7, 9, 3):
        monkeypatch.setattr(o, "SCAN_SCRATCH_BYTES", 4 * H * d * dv * places)
        outs, states = run(range(len(lens)))
        assert all(torch.equal(a, b) for a, b in zip(outs, together)) and torch.equal(states, end), places
    monkeypatch.undo()
    outs, states = run(range(len(lens)), deterministic=False)
    tol = 2e-6 if dtype == torch.float32 or form == "gated" else 2.0 ** -8
    for a, b in zip(outs + [states], together + [end]):
        assert float((a.double() - b.double()).norm()) <= tol * float(b.double().norm())


@pytest.mark.parametrize("what", ["vector state", "min gru", "latent attention"])
def test_a_deterministic_sets_short_runs_depend_on_no_other_sequence(what):
    """Runs too short for the forms that long ones take, alone and beside long ones: the same bits."""
    from supersonic_b200.csrc.fast_sets import FastKernels
    from test_sotavik_kernels_gpu import latent_case
    ks, lens, slots, C, H, dk, dv = FastKernels(deterministic=True), [30, 3, 300, 64, 2, 129], [3, 0, 6, 1, 5, 2], 128, 4, 48, 32
    T = sum(lens)
    gates, z_bias, x_bias, rate = rnd(T, 2 * C, seed=1), rnd(C, seed=2), rnd(C, seed=3), -torch.rand(C, device=DEV)
    u, y, proj = (rnd(T, w, seed=w + i, dtype=torch.bfloat16) for i, w in enumerate((C, C, 3 * C)))
    state0 = rnd(7, C, seed=7)

    def run(which):
        take = torch.cat([torch.arange(sum(lens[:i]), sum(lens[:i + 1])) for i in which]).to(DEV)
        batch, state = step_of([lens[i] for i in which], [slots[i] for i in which]), state0.clone()
        out = torch.full((len(take), H * dv if what == "latent attention" else C), math.nan, dtype=torch.bfloat16, device=DEV)
        if what == "vector state":
            ks.gated_unit_scan(gates[take], z_bias, x_bias, rate, u[take], y[take], z_bias, state, batch, out, 64)
        elif what == "min gru":
            ks.mingru_scan(proj[take], z_bias, x_bias, state, batch, out, C)
        else:
            new, past = [lens[i] for i in which], 170
            cache, batch, store, table, q, rows = latent_case([n + past for n in new], new, H, dk, dv, seed=5)
            for i, at in zip(which, [sum(new[:j]) for j in range(len(new))]):       # a sequence's own rows, whatever its place
                own = rnd(lens[i] + past, dk, seed=50 + i, dtype=torch.bfloat16)
                pages = table[batch.seq_slot[which.index(i)].long(), : -(-(lens[i] + past) // 64)].long()
                for j, page in enumerate(pages.tolist()):
                    piece = own[64 * j:64 * j + 64]
                    store[page, 0, : piece.shape[0]] = piece
                q[at:at + lens[i]] = rnd(lens[i], H * dk, seed=90 + i, dtype=torch.bfloat16)
            ks.latent_attention(q, store, batch, table, out, H, dv, dk - dv, 6, None, dk ** -0.5, None)
        assert bool(torch.isfinite(out.float()).all())
        return list(out.split([lens[i] for i in which])), state
    together, end = run(list(range(len(lens))))
    for group in ([0], [1], [4], [3], [0, 1], [1, 4], [5, 0], [2, 4]):
        outs, states = run(group)
        for i, out in zip(group, outs):
            assert torch.equal(out, together[i]) and torch.equal(states[slots[i]], end[slots[i]]), (group, i)


@pytest.mark.parametrize("kind", ["window", "pooled", "all", "sigmoid"])
@pytest.mark.parametrize("dim", [128, 64])
def test_a_cluster_of_blocks_shares_a_decode_steps_pages(kind, dim):
    """Every size of cluster against one block a (sequence, kv head), on sequences of one token, of fewer pages than blocks,
    of a window's edge and of many pages: float32 sums of a row merged in another order, then one rounding to bfloat16."""
    lens, n_q, n_kv = [1, 63, 64, 65, 130, 517, 700], 6, 2
    B, pages = len(lens), sum((n + 63) // 64 for n in lens)
    perm = torch.randperm(pages + 2, generator=torch.Generator().manual_seed(dim)).to(torch.int32)
    table, ptable, at = torch.zeros(B, 16, dtype=torch.int32), torch.arange(B, dtype=torch.int32)[:, None].repeat(1, 2), 0
    for b, n in enumerate(lens):
        table[b, :(n + 63) // 64] = perm[at:at + (n + 63) // 64]
        at += (n + 63) // 64
    k, v = (rnd(pages + 2, n_kv, 64, dim, seed=s, dtype=torch.bfloat16) for s in (1, 2))
    pk, pv = (rnd(B, n_kv, 64, dim, seed=s, dtype=torch.bfloat16) for s in (3, 4))
    q = rnd(B, n_q * dim, seed=5, dtype=torch.bfloat16)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    cu, start, slots, table, ptable = i32(list(range(B + 1))), i32([n - 1 for n in lens]), i32(list(range(B))), table.to(DEV), ptable.to(DEV)
    gate, sinks = rnd(B, n_q, seed=6, dtype=torch.bfloat16), rnd(n_q, seed=7)
    cos, sin = torch.cos(rnd(800, dim // 2, seed=8)), torch.sin(rnd(800, dim // 2, seed=8))

    def run(cluster):
        out = torch.full((B, n_q * dim), 9.0, device=DEV, dtype=torch.bfloat16)
        if kind == "sigmoid":
            ops().sigmoid_attention_mma(q, k, v, cu, start, slots, table, sinks, out, 1, n_q, n_kv, dim, dim, 6, 256, None,
                                        dim ** -0.5, split=True, cluster=cluster)
            return out.float()
        pooled = (pk, pv, ptable) if kind == "pooled" else None
        ops().window_attention_mma(q, k, v, table, pooled, cu, start, slots, out, 1, n_q, n_kv, dim, dim, 6,
                                   None if kind == "all" else 128, 3 if kind == "window" else 0, 16 if pooled else 0, dim ** -0.5,
                                   30.0, sinks if kind != "pooled" else None, cos if pooled else None, sin if pooled else None,
                                   False, split=True, gate=gate, cluster=cluster)
        return out.float()
    one = run(1)
    for cluster in (2, 3, 4, 8):
        got = run(cluster)
        # a value next to a rounding boundary may go either way: one step of bfloat16, 2^-8 of its size
        assert bool(((got - one).abs() <= 2.0 ** -7 * one.abs() + 1e-6).all()), cluster


@pytest.mark.parametrize("dim,vdim,n_q,n_kv,n_v", [(128, 128, 16, 4, 4), (64, 64, 32, 8, 8), (64, 128, 40, 20, 10), (128, 64, 3, 1, 1)])
@pytest.mark.parametrize("norm,rot,interleaved", [("head", 64, False), ("row", 32, True), (None, 0, False), ("head", 16, False)])
@pytest.mark.parametrize("T", [7, 128, 129, 300])
def test_rows_prepared_a_warp_a_head(dim, vdim, n_q, n_kv, n_v, norm, rot, interleaved, T):
    """Against the kernel that takes any width (which rows at an odd address still get): queries, cached keys and values, and
    the pooled rows of tokens that end a run; float32 in between, so one step of bfloat16 apart at the most."""
    pool = 16 if n_v == n_kv and T == 7 else 0
    width, positions = (n_q + n_kv) * dim + n_v * vdim, [0, 15, 63, 64, 127, 200, 31] if T == 7 else [t % 250 for t in range(T)]
    rows = rnd(T, width + 8, seed=dim + n_q, dtype=torch.bfloat16)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    pos, slots = i32(positions), i32([0, 1, 2, 3, 4, 5, -1] if T == 7 else [t // 250 for t in range(T)])
    table = torch.arange(6 * 4, dtype=torch.int32, device=DEV).view(6, 4)
    ptable = torch.arange(6, dtype=torch.int32, device=DEV).view(6, 1)
    qw, kw = (rnd(dim if norm == "head" else n * dim, seed=n) + 1.0 for n in (n_q, n_kv))
    cos, sin = (f(rnd(256, rot // 2, seed=5)) for f in (torch.cos, torch.sin)) if rot else (None, None)
    vcos, vsin = (f(rnd(256, vdim // 2, seed=6)) for f in (torch.cos, torch.sin))
    mix = (rnd(T, n_v * vdim, seed=9, dtype=torch.bfloat16), 0.3)
    got = []
    for odd in (True, False):
        qkv = rows.clone()[:, 2:2 + width] if odd else rows[:, 2:2 + width].contiguous()
        k, v = (rnd(24, n, 64, d, seed=n, dtype=torch.bfloat16) for n, d in ((n_kv, dim), (n_v, vdim)))
        pk, pv = (torch.zeros(6, n_kv, 64, d, device=DEV, dtype=torch.bfloat16) for d in (dim, vdim))
        ops().qkv_prepare(qkv, qw if norm else None, kw if norm else None, norm, 1e-5, cos, sin, rot, interleaved, vcos, vsin,
                          interleaved, pos, slots, table, k, v, n_q, n_kv, dim, vdim, 6, pooled=(pk, pv, ptable) if pool else None,
                          pool=pool, n_v=n_v, v_mix=mix, q_temp=(0.2, 8))
        got.append([x.float() for x in (qkv[:, : n_q * dim], k, v, pk, pv)])
    for a, b in zip(*got):
        assert bool(((a - b).abs() <= 2.0 ** -7 * a.abs() + 1e-5).all())
    if pool:                                                        # the tokens at 15, 63 and 127 end a run
        assert (got[1][3].abs().sum((1, 2, 3)) > 0).tolist() == [False, True, True, False, True, False]


@pytest.mark.parametrize("rot", [2, 6, 64])
def test_coordinates_beside_an_interleaved_rotation_stay_as_they_are(rot):
    """Heads of 128 of which a few leading coordinates turn in pairs: an infinity in the others stays where it is and spreads to
    no neighbour, in queries and in cached keys."""
    T, dim = 3, 128
    qkv = rnd(T, 3 * dim, seed=rot, dtype=torch.bfloat16)
    qkv[:, [rot + 1, rot + 8, dim + rot + 1]] = math.inf
    rows = qkv.clone()
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    cos, sin = torch.cos(rnd(64, rot // 2, seed=1)), torch.sin(rnd(64, rot // 2, seed=1))
    k, v = (torch.zeros(1, 1, 64, dim, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    ops().qkv_prepare(qkv, None, None, None, 1e-5, cos, sin, rot, True, None, None, False, i32([5, 6, 7]), i32([0, 0, 0]), i32([[0]]),
                      k, v, 1, 1, dim, dim, 6)
    assert torch.equal(qkv[:, rot:dim], rows[:, rot:dim]) and torch.equal(k[0, 0, 5:8, rot:], rows[:, dim + rot:2 * dim])
    assert torch.equal(v[0, 0, 5:8], rows[:, 2 * dim:]) and bool(torch.isfinite(qkv[:, :rot].float()).all())


@pytest.mark.parametrize("m,n,k", [(1, 8, 64), (31, 40, 128), (33, 72, 64), (129, 264, 192), (257, 1000, 128), (300, 256, 512),
                                   (8, 96, 64), (41, 96, 128)])
@pytest.mark.parametrize("tile", [64, 128, 256, "pair"])
def test_products_leave_in_whole_rows(m, n, k, tile):
    """Every way out of the tcgen05 product at ragged edges: the float32 sums stored, the same added to what is there (one
    rounding, whoever adds), the same rounded to bfloat16; nothing beside the result is touched."""
    o = ops()
    tile = o.TC_TILE_PAIR if tile == "pair" else tile
    a, w, c = rnd(m, k, seed=m, dtype=torch.bfloat16), rnd(n, k, seed=n, dtype=torch.bfloat16), rnd(m, n, seed=k)
    wide = [torch.full((m + 1, n + 8), 5.0, device=DEV, dtype=t) for t in (torch.float32, torch.float32, torch.bfloat16)]
    sums, added, rounded = (x[:m, :n] for x in wide)
    added.copy_(c)
    for out, mode in ((sums, o.TC_STORE), (added, o.TC_ACCUMULATE), (rounded, o.TC_STORE)):
        o.gemm_tc(a, w, out, mode, tile_n=tile)
    o.check_device_errors(torch.device(DEV))
    want = a.double() @ w.double().t()
    # k products of float32 sums: k 2^-24 of the sum of their sizes
    assert bool(((sums.double() - want).abs() <= k * 2.0 ** -24 * (a.double().abs() @ w.double().abs().t()) + 1e-30).all())
    assert torch.equal(added, c + sums) and torch.equal(rounded, sums.to(torch.bfloat16))
    assert all(bool((x[m] == 5.0).all() and (x[:, n:] == 5.0).all()) for x in wide)


@pytest.mark.parametrize("tile", [256, "pair"])
def test_rows_of_no_slot_have_no_position(tile):
    """The projection that rotates and appends skips rows with a negative slot, whatever their position says: one far outside the
    rotation tables is not looked up, and the other rows, in the same warps, are as they are without them."""
    o, rows, hd, n_q, n_kv = ops(), 140, 64, 2, 1
    tile = o.TC_TILE_PAIR if tile == "pair" else tile
    a, w = rnd(rows, 128, seed=1, dtype=torch.bfloat16), rnd((n_q + 2 * n_kv) * hd, 128, seed=2, scale=0.1, dtype=torch.bfloat16)
    cos, sin = torch.cos(rnd(256, hd // 2, seed=3)), torch.sin(rnd(256, hd // 2, seed=3))
    table = torch.arange(4, dtype=torch.int32, device=DEV).view(1, 4)
    dead = torch.arange(rows, device=DEV) % 3 == 1
    got = []
    for outside in (False, True):
        pos = torch.arange(rows, dtype=torch.int32, device=DEV)
        slot = torch.where(dead, -1, 0).to(torch.int32)
        if outside:
            pos[dead] = 1 << 30
        q = torch.full((rows, n_q * hd), 5.0, dtype=torch.bfloat16, device=DEV)
        k, v = (torch.full((4, n_kv, 64, hd), 5.0, dtype=torch.bfloat16, device=DEV) for _ in range(2))
        o.gemm_tc_rope_append(a, w, q, cos, sin, pos, slot, table, k, v, n_q, n_kv, hd, 6, tile_n=tile)
        o.check_device_errors(torch.device(DEV))
        assert bool((q[dead] == 5.0).all()) and bool((q[~dead] != 5.0).any(1).all())
        got.append((q, k, v))
    assert all(torch.equal(x, y) for x, y in zip(*got))


@pytest.mark.parametrize("rows", [129, 300, 1024])
def test_a_chain_of_dependent_launches_reads_what_was_written(rows):
    """Norm, product, product into the stream, attention's preparation: launched as programmatic dependents of one another or
    one after the other, many times over the same buffers, the same bits."""
    o, n = ops(), 512
    w1, w2 = (rnd(n, n, seed=s, scale=n ** -0.5, dtype=torch.bfloat16) for s in (1, 2))
    gain, pos = torch.ones(n, device=DEV), torch.arange(rows, dtype=torch.int32, device=DEV)
    slot, table = torch.zeros(rows, dtype=torch.int32, device=DEV), torch.arange(16, dtype=torch.int32, device=DEV).view(1, 16)
    angle = rnd(1024, 32, seed=3)
    cos, sin = torch.cos(angle), torch.sin(angle)
    got = []
    for pdl in (False, True):
        x, h, y = rnd(rows, n, seed=rows), torch.empty(rows, n, dtype=torch.bfloat16, device=DEV), torch.empty(rows, n, dtype=torch.bfloat16, device=DEV)
        k, v = (torch.zeros(16, 2, 64, 64, dtype=torch.bfloat16, device=DEV) for _ in range(2))
        torch.cuda.synchronize()
        for turn in range(30):
            tile = (64, 128, 256, o.TC_TILE_PAIR)[turn % 4]
            o.rmsnorm_vec(x, gain, 1e-5, h, pdl=pdl)
            o.gemm_tc(h, w1, y, tile_n=tile, pdl=pdl)
            o.rope_append_vec(y, cos, sin, pos, slot, table, k, v, 4, 2, 64, 6, pdl=pdl)
            o.gemm_tc(y, w2, x, o.TC_ACCUMULATE, tile_n=tile, pdl=pdl)
        o.check_device_errors(torch.device(DEV))
        got.append((x.clone(), y.clone(), k.clone(), v.clone()))
    assert all(torch.equal(a, b) for a, b in zip(*got))


@pytest.mark.parametrize("lens,starts,hd", [([129], [0], 64), ([1, 200, 64, 5], [70, 0, 64, 300], 128), ([700, 324], [0, 9], 128)])
def test_a_chain_of_a_prompts_layer_reads_what_was_written(lens, starts, hd):
    """A prompt's layer as a step launches it: the projection that rotates and appends, attention, the products of the gated
    unit, of an activation and into the stream, as programmatic dependents of one another or one after the other: the same bits."""
    o, rows, n_q, n_kv = ops(), sum(lens), 4, 2
    n, width = n_q * hd, (n_q + 2 * n_kv) * hd
    w_qkv, w_o, w_gate, w_down, w_act = (rnd(a, b, seed=s, scale=b ** -0.5, dtype=torch.bfloat16) for s, (a, b) in
                                         enumerate([(width, n), (n, n), (2 * n, n), (n, n), (n, n)]))
    gain, angle = torch.ones(n, device=DEV), rnd(2048, hd // 2, seed=7)
    cos, sin = torch.cos(angle), torch.sin(angle)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    cu, start, seq_slot = i32([sum(lens[:i]) for i in range(len(lens) + 1)]), i32(starts), i32(list(range(len(lens))))
    pos = torch.cat([torch.arange(s, s + k) for s, k in zip(starts, lens)]).to(torch.int32).to(DEV)
    slot = torch.repeat_interleave(seq_slot, i32(lens).long())
    table = torch.arange(16 * len(lens), dtype=torch.int32, device=DEV).view(-1, 16)
    got = []
    for pdl in (False, True):
        x, (k, v) = rnd(rows, n, seed=rows), (rnd(16 * len(lens), n_kv, 64, hd, seed=s, dtype=torch.bfloat16) for s in (8, 9))
        h, q, att, z, y = (torch.zeros(rows, n, dtype=torch.bfloat16, device=DEV) for _ in range(5))
        torch.cuda.synchronize()
        for turn in range(20):
            wide = (256, o.TC_TILE_PAIR)[turn % 2]
            tile = (64, 128, 256, o.TC_TILE_PAIR)[turn % 4]
            o.rmsnorm_vec(x, gain, 1e-5, h, pdl=pdl)
            o.gemm_tc_rope_append(h, w_qkv, q, cos, sin, pos, slot, table, k, v, n_q, n_kv, hd, 6, tile_n=wide, pdl=pdl)
            o.attention_prefill_tc(q, k, v, cu, start, seq_slot, table, att, max(lens), n_q, n_kv, hd, 6, None, hd ** -0.5, pdl=pdl)
            o.gemm_tc(att, w_o, x, o.TC_ACCUMULATE, tile_n=tile, pdl=pdl)
            o.rmsnorm_vec(x, gain, 1e-5, h, pdl=pdl)
            if turn % 3:
                o.gemm_tc(h, w_gate, z, o.TC_SWIGLU, tile_n=tile, pdl=pdl)
            else:
                o.gemm_tc_gate(h, w_gate, z, ("gelu_tanh", 0.0), None, tile_n=tile, pdl=pdl)
            o.gemm_tc_act(z, w_act, y, "silu", 0.5, tile_n=tile, pdl=pdl)
            o.gemm_tc(y, w_down, x, o.TC_ACCUMULATE, tile_n=tile, pdl=pdl)
        o.check_device_errors(torch.device(DEV))
        got.append((x.clone(), q.clone(), k.clone(), v.clone(), att.clone()))
    assert all(bool(torch.isfinite(t.float()).all()) for t in got[0])
    assert all(torch.equal(a, b) for a, b in zip(*got))


@pytest.mark.parametrize("rows", [129, 300])
def test_a_chain_of_products_in_parts_reads_what_was_written(rows):
    """Products whose K is cut into parts, rounded and cleared, the sums used again by the next: chained or not, each turn's
    result is that of its own inputs.  Parts add in any order: float32 sums of 1,024 products, then one rounding."""
    o, n, k = ops(), 256, 1024
    w, back = rnd(n, k, seed=1, scale=k ** -0.5, dtype=torch.bfloat16), rnd(k, n, seed=2, scale=n ** -0.5, dtype=torch.bfloat16)
    for pdl in (False, True):
        sums, a, y = torch.zeros(rows, n, device=DEV), rnd(rows, k, seed=rows, dtype=torch.bfloat16), torch.empty(rows, n, dtype=torch.bfloat16, device=DEV)
        torch.cuda.synchronize()
        seen = []
        for turn in range(12):
            o.gemm_tc(a, w, sums, o.TC_ACCUMULATE, tile_n=128, splits=4, pdl=pdl)
            o.round_and_clear(sums, y, pdl=pdl, act="silu" if turn % 2 else None)
            a, before = torch.empty_like(a), a
            o.gemm_tc(y, back, a, tile_n=128, pdl=pdl)
            seen.append((before, y.clone(), a))
        o.check_device_errors(torch.device(DEV))
        assert bool((sums == 0).all())
        for turn, (x, y_, a_) in enumerate(seen):
            want = x.double() @ w.double().t()
            want = torch.nn.functional.silu(want) if turn % 2 else want
            bound = k * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t()) + 2.0 ** -8 * want.abs() + 1e-30
            assert bool(((y_.double() - want).abs() <= bound).all()), (pdl, turn)
            want = y_.double() @ back.double().t()
            bound = n * 2.0 ** -24 * (y_.double().abs() @ back.double().abs().t()) + 2.0 ** -8 * want.abs() + 1e-30
            assert bool(((a_.double() - want).abs() <= bound).all()), (pdl, turn)


@pytest.mark.parametrize("width", [8, 2048, 516, 1030])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_sums_of_a_few_rows_in_their_order(width, dtype):
    """Experts' rows and streams added up four columns a thread (or, in rows that are not whole pieces, one): the same chain
    of multiply-adds, against the rows at an odd address."""
    for tokens, top in ((1, 1), (5, 6), (300, 4), (3, 9)):
        y, w, res = rnd(tokens * top, width, seed=top, dtype=dtype), rnd(tokens, top, seed=tokens), rnd(tokens, width, seed=3)
        want, got = res.clone(), res.clone()
        ops().expert_combine(want, off_by_one(y), w, top)
        ops().expert_combine(got, y, w, top)
        assert torch.equal(got, want)
        if dtype == torch.float32:
            streams = rnd(top, tokens, width, seed=5)
            one, other = torch.empty(tokens, width, device=DEV), torch.empty(tokens, width, device=DEV)
            ops().stream_mix(off_by_one(streams), w[0].contiguous(), top, one)
            ops().stream_mix(streams, w[0].contiguous(), top, other)
            assert torch.equal(one, other)


@pytest.mark.parametrize("n_seqs,longest,n_q,n_kv,hd,window",
                         [(600, 90, 2, 1, 64, None), (40, 700, 6, 2, 128, None), (150, 300, 3, 1, 64, 100), (150, 300, 3, 3, 128, 65),
                          (3, 400, 8, 2, 128, None), (2, 700, 5, 1, 64, None), (37, 512, 8, 4, 64, None)])
def test_prompt_attention_over_many_units(n_seqs, longest, n_q, n_kv, hd, window):
    """Blocks that stay for many units of a ragged batch, more sequences than a launch's table holds, sequences without a slot or
    without tokens, one tile a unit and two.  Probabilities are rounded to bfloat16 (2^-9 of the largest value), and so is the
    output (2^-9 again)."""
    o, g = ops(), torch.Generator().manual_seed(n_seqs + longest)
    lens, starts = torch.randint(1, longest + 1, (n_seqs,), generator=g), torch.randint(0, 200, (n_seqs,), generator=g)
    lens[0], starts[0] = longest, 0
    lens[n_seqs // 2] = 0 if n_seqs > 10 else 1
    pages = (longest + 200 + 63) // 64
    slot = torch.arange(n_seqs, dtype=torch.int32)
    if n_seqs > 10:
        slot[3::7] = -1
    table = torch.randperm(n_seqs * pages, generator=g).to(torch.int32).view(n_seqs, pages).to(DEV)
    k, v = (rnd(n_seqs * pages, n_kv, 64, hd, seed=s, dtype=torch.bfloat16) for s in (1, 2))
    cu = torch.cat([torch.zeros(1, dtype=torch.int64), lens.cumsum(0)])
    rows = int(cu[-1])
    q = rnd(rows, (n_q + 2 * n_kv) * hd, seed=3, dtype=torch.bfloat16)
    out = torch.full((rows, n_q * hd), 7.0, dtype=torch.bfloat16, device=DEV)
    o.attention_prefill_tc(q, k, v, cu.to(torch.int32).to(DEV), starts.to(torch.int32).to(DEV), slot.to(DEV), table, out, longest,
                           n_q, n_kv, hd, 6, window, hd ** -0.5)
    o.check_device_errors(torch.device(DEV))
    for b in range(n_seqs):
        r0, n, s = int(cu[b]), int(lens[b]), int(starts[b])
        mine = out[r0:r0 + n].view(n, n_q, hd)
        if slot[b] < 0:
            assert bool((mine == 7.0).all())
            continue
        keys, values = (c[table[b].long()].transpose(0, 1).reshape(n_kv, -1, hd)[:, :s + n].double().repeat_interleave(n_q // n_kv, 0)
                        for c in (k, v))
        score = torch.einsum("nhd,hkd->hnk", q[r0:r0 + n, :n_q * hd].view(n, n_q, hd).double(), keys) * hd ** -0.5
        at, key = torch.arange(s, s + n, device=DEV)[:, None], torch.arange(s + n, device=DEV)[None]
        seen = (key <= at) & (key > at - window if window else key >= 0)
        want = torch.softmax(score.masked_fill(~seen, -math.inf), -1) @ values
        assert n == 0 or float((mine.double() - want.transpose(0, 1)).abs().max()) <= 2.0 ** -8 * 1.05 * float(values.abs().max())


@pytest.mark.parametrize("n_q,n_kv,hd,window,n,start", [(3, 1, 64, 65, 300, 0), (1, 1, 128, 65, 260, 0), (5, 1, 64, 100, 700, 30), (6, 2, 128, 129, 400, 200),
                                                        (3, 1, 64, None, 300, 0)])
def test_windowed_prompt_attention_is_the_same_bits_in_every_batch(n_q, n_kv, hd, window, n, start):
    """An odd number of query heads a kv head: the second tile of a unit may lie in the next row tile.  A prompt alone (one tile
    a unit) and among others that make enough units for two."""
    o, pages = ops(), (n + start + 63) // 64
    others = o.sm_count() // n_kv                                   # at least two units each: more than one a multiprocessor
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    k, v = (rnd(pages, n_kv, 64, hd, seed=s, dtype=torch.bfloat16) for s in (1, 2))
    q = rnd(n, (n_q + 2 * n_kv) * hd, seed=3, dtype=torch.bfloat16)

    def run(seqs):                                                  # the same prompt in every place, over the same pages
        out = torch.empty(seqs * n, n_q * hd, dtype=torch.bfloat16, device=DEV)
        o.attention_prefill_tc(q.repeat(seqs, 1), k, v, i32([i * n for i in range(seqs + 1)]), i32([start] * seqs), i32([0] * seqs),
                               i32([list(range(pages))]), out, n, n_q, n_kv, hd, 6, window, hd ** -0.5)
        o.check_device_errors(torch.device(DEV))
        return out.view(seqs, n, -1)
    alone, among = run(1)[0], run(others + 1)
    assert all(torch.equal(alone, row) for row in among)


@pytest.mark.parametrize("n", [0, 1, 128, 129, 960, 961, 1920, 2500])
@pytest.mark.parametrize("n_before", [0, 1, 300])
def test_a_steps_integers_come_in_their_places(n, n_before):
    """Around the sizes of one launch's arguments and of one launch, with and without a device tensor in front; what lies beside
    the destination stays as it is."""
    values = torch.arange(n, dtype=torch.int32).add(7).numpy()
    before = torch.arange(n_before, dtype=torch.int32, device=DEV).sub(500) if n_before else None
    room = torch.full((n + n_before + 8,), -9, dtype=torch.int32, device=DEV)
    ops().put_ints(values, room[4:4 + n + n_before], before=before)
    values[:] = 0                                                   # taken at the call
    want = torch.cat([torch.full((4,), -9), torch.arange(n_before) - 500, torch.arange(n) + 7, torch.full((4,), -9)])
    assert torch.equal(room.cpu().long(), want)


@pytest.mark.parametrize("n_states", [0, 1, 96, 97, 200])
def test_an_opened_sequence_starts_from_zeros(n_states):
    """No state rows, a launch's worth of them and more, rows from one word to more than a block's share; other slots keep theirs."""
    rng = torch.arange(5, dtype=torch.int64, device=DEV)
    states = [torch.full((5, 1 + 37 * i if i != 1 else 300001), 3.0, device=DEV) for i in range(n_states)]
    ops().open_sequence(rng, 2, -1234567890123456789, states)
    assert rng.tolist() == [0, 1, -1234567890123456789, 3, 4]
    keep = torch.tensor([0, 1, 3, 4], device=DEV)
    assert all(bool((t[2] == 0).all()) and bool((t[keep] == 3).all()) for t in states)
    with pytest.raises(ops().KernelError, match="slot"):
        ops().open_sequence(rng, 5, 1, states)


def test_the_host_and_the_kernel_agree_on_the_integers_a_launch_takes():
    from supersonic_b200.csrc.build import load_library
    assert load_library("step_inputs").ssb_put_ints_most() == ops().PUT_INTS_MOST


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n_q,n_kv,hd,rot,interleaved,T", [(6, 3, 64, 64, False, 700), (5, 1, 24, 8, True, 1400), (17, 2, 32, 0, False, 500)])
def test_rotation_of_many_tokens_is_that_of_a_few(dtype, n_q, n_kv, hd, rot, interleaved, T):
    """So many tokens that a block takes all of one's heads, and the same tokens seven at a time (eight heads a block)."""
    o = ops()
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    pos, slot = i32([t // 2 for t in range(T)]), i32([-1 if t % 50 == 7 else t % 2 for t in range(T)])
    pages = T // 128 + 1
    table = torch.randperm(2 * pages, generator=torch.Generator().manual_seed(T)).to(torch.int32).view(2, pages).to(DEV)
    cos, sin = rnd(T // 2 - 3, rot // 2, seed=5), rnd(T // 2 - 3, rot // 2, seed=6)
    qkv = rnd(T, (n_q + 2 * n_kv) * hd, seed=3, dtype=dtype)
    got = []
    for step in (T, 7):
        x, k, v = qkv.clone(), torch.zeros(2 * pages, n_kv, 64, hd, dtype=dtype, device=DEV), torch.zeros(2 * pages, n_kv, 64, hd, dtype=dtype, device=DEV)
        for a in range(0, T, step):
            b = slice(a, a + step)
            o.rope_append(x[b], cos if rot else None, sin if rot else None, pos[b], slot[b], table, k, v, n_q, n_kv, hd, rot, 6,
                          interleaved=interleaved)
        got.append((x, k, v))
    assert all(torch.equal(a, b) for a, b in zip(*got)) and not torch.equal(got[0][1], torch.zeros_like(got[0][1]))


@pytest.mark.parametrize("H,d,dv,B", [(4, 256, 512, 40), (2, 256, 512, 3), (4, 128, 256, 30), (4, 128, 256, 2)])
def test_gated_scan_of_one_token_is_as_close_to_64_bits_as_the_walk(H, d, dv, B):
    """In wide and in narrow blocks.  N random products in chains of n that meet in a tree of L levels are off by about
    sqrt(N (n / 2 + L)) roundings: chains of 16 or 8 and 4 or 5 levels here, of 4 and 6 levels in the walk of 256 rows, at most
    sqrt(12 / 8) = 1.22 times as far.  (Chains of 32 and one over the parts were 1.36 to 1.45 times as far.)"""
    proj, z, bias = rnd(B, 2 * H * d + H * dv, seed=d, dtype=torch.bfloat16), rnd(B, H * d, seed=1), rnd(H * d, seed=2) + 3.0
    state0, i32 = rnd(B, H * d * dv, seed=3), torch.arange(B + 1, dtype=torch.int32, device=DEV)
    decay = torch.sigmoid(z.double() + bias.double()).pow(1 / 16.0).view(B, H, d, 1)
    q, k, v = (proj[:, a:b].double() for a, b in ((0, H * d), (H * d, 2 * H * d), (2 * H * d, 2 * H * d + H * dv)))
    S = decay * state0.double().view(B, H, d, dv) + k.view(B, H, d, 1) * v.view(B, H, 1, dv)
    want, off = torch.einsum("bhd,bhdv->bhv", q.view(B, H, d), S).reshape(B, -1), []
    for form in (1, 3):
        out = torch.zeros(B, H * dv, device=DEV)
        ops().gated_linear_scan(proj, 0, H * d, 2 * H * d, z.clone(), bias, 16.0, 1.0, state0.clone(), i32, i32[:B], out, H, d, dv, form=form)
        off.append(float((out.double() - want).norm() / want.norm()))
    assert off[1] <= 1.25 * off[0], off
