"""Each CUDA kernel alone against its plain statement (tests/reference_kernels.py), at sizes other
than the tiny models': widths and vocabularies that are no power of two, head sizes in steps of 16,
odd group sizes, and inputs made so that a fault in an index shows (one key that stands out among
hundreds, the window's edge, the slot of the cache)."""
import math
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from reference_kernels import ReferenceKernels
from cima_b200.cache.kv import LayerKV

pytestmark = pytest.mark.gpu

REF = ReferenceKernels(compute=torch.float64)
DT = {"float32": torch.float32, "bfloat16": torch.bfloat16}
# one rounding to the output dtype of values of magnitude about 1, plus summation error
TOL = {"float32": 2e-5, "bfloat16": 1.6e-2}


@pytest.fixture(scope="module")
def K():
    from cima_b200.kernels import Kernels
    return Kernels(verbose=False)


def g(*shape, dtype=torch.float32, seed=0, scale=1.0):
    gen = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=gen) * scale).to(dtype)


def err(a, b):
    return (a.double().cpu() - b.double().cpu()).abs().max().item()


# ---------------------------------------------------------------------------- elementwise
@pytest.mark.parametrize("wdtype", ["float32", "bfloat16"])
def test_embed(K, wdtype):
    V, H = 777, 200
    table = g(V, H, dtype=DT[wdtype])
    ids = torch.tensor([0, 776, 5, 5, 300], dtype=torch.int32)
    x = torch.full((5, H), -7.0, device="cuda")
    K.embed(ids.cuda(), table.cuda(), x, 1.0)
    assert torch.equal(x.cpu(), table[ids.long()].float())


@pytest.mark.parametrize("odtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("H,eps", [(200, 3e-6), (3584, 1e-6), (1, 1e-5), (1000, 1e-2)])
def test_rmsnorm(K, odtype, H, eps):
    x, w = g(13, H, seed=1, scale=3.0), 1 + g(H, seed=2, scale=0.1)
    out = torch.empty(13, H, dtype=DT[odtype], device="cuda")
    K.rmsnorm(x.cuda(), w.cuda(), eps, out)
    want = torch.empty(13, H, dtype=torch.float64)
    REF.rmsnorm(x, w, eps, want)
    assert err(out, want) <= TOL[odtype] * 4


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_swiglu_and_residual_and_gather(K, dtype):
    T, I = 37, 328
    gu = g(T, 2 * I, dtype=DT[dtype], seed=3, scale=2.0)
    out = torch.empty(T, I, dtype=DT[dtype], device="cuda")
    for code in (0, 1, 2, 3):                           # the gate's activation: SiLU, GELU (tanh, erf), ReLU
        K.swiglu(gu.cuda(), out, code)
        want = torch.empty(T, I, dtype=torch.float64)
        REF.swiglu(gu, want, code)
        assert err(out, want) <= TOL[dtype] * 4, code
    x, d = g(T, I, seed=4), g(T, I, dtype=DT[dtype], seed=5)
    xg = x.cuda()
    K.add_residual(xg, d.cuda())
    assert torch.equal(xg.cpu(), x + d.float())
    rows = torch.tensor([36, 0, 0, 17], dtype=torch.int32)
    picked = torch.empty(4, I, device="cuda")
    K.gather_rows(xg, rows.cuda(), picked)
    assert torch.equal(picked.cpu(), xg.cpu()[rows.long()])


# ---------------------------------------------------------------------------- matrix products
@pytest.mark.parametrize("M,N,K_", [(1, 192, 448), (7, 1000, 333), (130, 65, 17), (64, 64, 64)])
@pytest.mark.parametrize("combo", [("float32", "float32", "float32"), ("bfloat16", "float32", "bfloat16"),
                                   ("bfloat16", "bfloat16", "float32")])
def test_linear_plain(K, M, N, K_, combo):
    a, w, b = g(M, K_, dtype=DT[combo[0]], seed=1), g(N, K_, dtype=DT[combo[1]], seed=2, scale=0.1), g(N, seed=3)
    # guard columns around the output prove that nothing is written outside it
    # (the reference's sentinel check, src/selftest.rs:803, :837-850)
    out = torch.full((M, N), -777.0, dtype=DT[combo[2]], device="cuda")
    K.linear_plain(a.cuda(), w.cuda(), b.cuda(), out)
    want = a.double() @ w.double().t() + b.double()
    assert err(out, want) <= TOL[combo[2]] * max(1.0, want.abs().max().item())
    if combo[2] == "float32":
        acc = torch.ones(M, N, device="cuda")
        K.linear_plain(a.cuda(), w.cuda(), None, acc, accumulate=True)
        assert err(acc, 1 + a.double() @ w.double().t()) <= 2e-5 * max(1.0, want.abs().max().item())


@pytest.mark.parametrize("rows", [1, 5, 8])
@pytest.mark.parametrize("N,K_", [(300, 200), (65, 7), (1000, 3584)])
def test_linear_plain_rows_are_independent(K, rows, N, K_):
    """The same bits for a row whether it comes among 70 (the tiled kernel) or among at most 8 (the kernel of
    the decode steps, one thread per output feature): both add the products of an output in ascending k."""
    a, w, b = g(70, K_, seed=1), g(N, K_, seed=2), g(N, seed=3)
    full = torch.empty(70, N, device="cuda")
    K.linear_plain(a.cuda(), w.cuda(), b.cuda(), full)
    few = torch.empty(rows, N, device="cuda")
    K.linear_plain(a[33:33 + rows].contiguous().cuda(), w.cuda(), b.cuda(), few)
    assert torch.equal(full[33:33 + rows], few)
    acc_full, acc_few = torch.ones(70, N, device="cuda"), torch.ones(rows, N, device="cuda")
    K.linear_plain(a.cuda(), w.cuda(), None, acc_full, accumulate=True)
    K.linear_plain(a[33:33 + rows].contiguous().cuda(), w.cuda(), None, acc_few, accumulate=True)
    assert torch.equal(acc_full[33:33 + rows], acc_few)


@pytest.mark.parametrize("N,K_", [(129, 256), (127, 512), (128, 513), (127, 516), (896, 4864), (20000, 896), (260, 1000), (130, 1021), (40, 4864), (2367, 200), (2377, 510),
                                  (9473, 72), (9479, 37)])
def test_linear_float32_the_same_bits_from_every_kernel(K, N, K_):
    """Rows 1 to 8 (a warp a range of k), 9 to 32, 33 to 64, 65 and more (tiles of 32, 64 and 128 rows; shared by a cluster where a
    product has few tiles, alone where it has many): one order of the sums, so one result; sizes around the tiles' edges, sums of one
    range of k (up to 512; one, two and eight warps a block with 8 features each) and of eight, ranges that end early, rows whose bytes are no multiple of 16.  Tolerance: a range's steps (K, or
    at most K / 8 + 15) and the eight ranges', each half an ulp of a sum that stays below the sum of the magnitudes."""
    M = 200
    a, w, b = g(M, K_, seed=4), g(N, K_, seed=5, scale=0.1), g(N, seed=6)
    want = a.double() @ w.double().t() + b.double()
    full = torch.empty(M, N, device="cuda")
    K.linear_plain(a.cuda(), w.cuda(), b.cuda(), full)
    room = (K_ if K_ <= 512 else K_ / 8 + 23) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().t()).max().item()
    assert err(full, want) <= room
    for rows in (1, 2, 3, 4, 5, 6, 7, 8, 9, 32, 33, 64, 65, 128):
        part = torch.full((rows, N), -777.0, device="cuda")
        K.linear_plain(a[50:50 + rows].contiguous().cuda(), w.cuda(), b.cuda(), part)
        assert torch.equal(part, full[50:50 + rows]), rows
        acc, acc_full = torch.ones(rows, N, device="cuda"), torch.ones(M, N, device="cuda")
        K.linear_plain(a[50:50 + rows].contiguous().cuda(), w.cuda(), None, acc, accumulate=True)
        K.linear_plain(a.cuda(), w.cuda(), None, acc_full, accumulate=True)
        assert torch.equal(acc, acc_full[50:50 + rows]), rows


@pytest.mark.parametrize("rows", [1, 5, 8])
def test_linear_float32_by_a_matrix_that_the_kernel_before_it_wrote(K, rows):
    """A product whose matrix is the result of the product launched just before it, without waiting in between: the new matrix is
    read, not what stood there before; as weights (``linear_plain_of_weights``) once it is old."""
    N, K_ = 4096, 1024
    a, left, right = g(rows, K_, seed=1).cuda(), g(N, 64, seed=2).cuda(), g(K_, 64, seed=3, scale=0.1).cuda()
    w, out, again = torch.empty(N, K_, device="cuda"), torch.empty(rows, N, device="cuda"), torch.empty(rows, N, device="cuda")
    want = a.double() @ (left.double() @ right.double().t()).t()
    for _ in range(10):
        w.fill_(float("nan"))
        torch.cuda.synchronize()
        K.linear_plain(left, right, None, w)
        K.linear_plain(a, w, None, out)
        # float32 sums of 64 and of 1,024 products
        assert err(out, want) <= (64 + 1024 / 8 + 23) * 2.0 ** -24 * (a.double().abs() @ (left.double().abs() @ right.double().abs().t()).t()).max().item()
    torch.cuda.synchronize()
    K.linear_plain_of_weights(a, w, None, again)
    assert torch.equal(out, again)


@pytest.mark.parametrize("M", [1, 3, 7, 8])
@pytest.mark.parametrize("N,K_", [(200, 328), (1000, 192), (4608, 3584), (17, 8)])
def test_linear_skinny_modes(K, M, N, K_):
    from cima_b200.kernels import SK_ACCUM, SK_STORE, SK_STORE_F32, SK_SWIGLU
    a = g(M, K_, dtype=torch.bfloat16, seed=M)
    w = g(N, K_, dtype=torch.bfloat16, seed=N, scale=1.0 / math.sqrt(K_))
    b = g(N, seed=7)
    want = a.double() @ w.double().t()
    out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    K.linear_skinny(a.cuda(), w.cuda(), b.cuda(), out, SK_STORE)
    assert err(out, want + b.double()) <= TOL["bfloat16"] * 4
    out32 = torch.empty(M, N, device="cuda")
    K.linear_skinny(a.cuda(), w.cuda(), None, out32, SK_STORE_F32)
    assert err(out32, want) <= 1e-4
    x = g(M, N, seed=9)
    xg = x.cuda()
    K.linear_skinny(a.cuda(), w.cuda(), None, xg, SK_ACCUM)
    assert err(xg, x.double() + want) <= 1e-4
    if N % 2 == 0:
        I = N // 2
        gg, uu = want[:, :I], want[:, I:]
        for code in (0, 1, 2, 3):                       # the gate's activation: SiLU, GELU (tanh, erf), ReLU
            act = torch.empty(M, I, dtype=torch.bfloat16, device="cuda")
            K.linear_skinny(a.cuda(), w.cuda(), None, act, SK_SWIGLU, act=code)
            assert err(act, REF.gate_act(gg, code) * uu) <= TOL["bfloat16"] * 4, code
        with pytest.raises(Exception, match="activation code"):
            K.linear_skinny(a.cuda(), w.cuda(), None, act, SK_SWIGLU, act=9)


def test_linear_skinny_row_does_not_depend_on_batch(K):
    from cima_b200.kernels import SK_STORE_F32
    a, w = g(8, 448, dtype=torch.bfloat16, seed=1), g(1000, 448, dtype=torch.bfloat16, seed=2)
    full = torch.empty(8, 1000, device="cuda")
    K.linear_skinny(a.cuda(), w.cuda(), None, full, SK_STORE_F32)
    for m in (1, 2, 5, 7):
        part = torch.empty(m, 1000, device="cuda")
        K.linear_skinny(a[:m].contiguous().cuda(), w.cuda(), None, part, SK_STORE_F32)
        assert torch.equal(part, full[:m])


@pytest.mark.parametrize("I,K_", [(7104, 72), (7105, 200), (8960, 264), (9472, 136), (9473, 72)])
def test_linear_skinny_gated_around_one_wave_of_blocks(K, I, K_):
    """444, 445, 560, 592 and 593 tiles of 16 features: three and four blocks on each of 148 SMs, and one more, with the folded norm
    and without.  Tolerance: the result's rounding to bfloat16, 2^-8 of it, and float32 sums of up to 264 products before."""
    from cima_b200.kernels import SK_SWIGLU
    a, w = g(8, K_, dtype=torch.bfloat16, seed=I), g(2 * I, K_, dtype=torch.bfloat16, seed=1, scale=1.0 / math.sqrt(K_))
    ssq = torch.rand(8, 5, generator=torch.Generator().manual_seed(2))
    inv = 1.0 / torch.sqrt(ssq.double().sum(1, keepdim=True) / K_ + 1e-6)
    plain, folded, one = (torch.empty(m, I, dtype=torch.bfloat16, device="cuda") for m in (8, 8, 1))
    K.linear_skinny(a.cuda(), w.cuda(), None, plain, SK_SWIGLU)
    K.linear_skinny(a[6:7].contiguous().cuda(), w.cuda(), None, one, SK_SWIGLU)
    K.linear_skinny_norm(a.cuda(), ssq.cuda(), 1e-6, w.cuda(), None, folded, SK_SWIGLU)
    for got, f in ((plain, 1.0), (folded, inv)):
        z = f * (a.double() @ w.double().t())
        want = REF.gate_act(z[:, :I], 0) * z[:, I:]
        assert err(got, want) <= 2.0 ** -8 * (1 + 2.0 ** -6) * want.abs().max().item()
    assert torch.equal(one, plain[6:7])


def test_linear_skinny_refuses(K):
    from cima_b200.kernels import KernelError, SK_STORE
    a, w = g(9, 64, dtype=torch.bfloat16).cuda(), g(32, 64, dtype=torch.bfloat16).cuda()
    with pytest.raises(KernelError, match="at most 8"):
        K.linear_skinny(a, w, None, torch.empty(9, 32, dtype=torch.bfloat16, device="cuda"), SK_STORE)
    a, w = g(2, 12, dtype=torch.bfloat16).cuda(), g(32, 12, dtype=torch.bfloat16).cuda()
    with pytest.raises(KernelError, match="multiples of 8"):
        K.linear_skinny(a, w, None, torch.empty(2, 32, dtype=torch.bfloat16, device="cuda"), SK_STORE)


# ---------------------------------------------------------------------------- cache and attention
def make_kv(n_pages, nkv, page, hd, n_slots, width, ring, window, dtype, tables):
    """A layer's pages (filled with a large stale value) and block table, on the GPU and mirrored on the CPU."""
    storage = torch.full((n_pages, 2, nkv, page, hd), 50.0, dtype=dtype)
    table = torch.zeros(n_slots, width, dtype=torch.int32)
    for slot, pages in tables.items():
        table[slot, :len(pages)] = torch.tensor(pages, dtype=torch.int32)
    cpu = LayerKV(storage, table, page, ring, window, 0)
    gpu = LayerKV(storage.cuda(), table.cuda(), page, ring, window, 0)
    return cpu, gpu


def batch_of(seqs, device):
    """seqs: list of (slot, start_pos, n_tokens) -> the arrays the kernels take."""
    row_pos, row_seq, first = [], [], [0]
    for i, (slot, start, n) in enumerate(seqs):
        row_pos += list(range(start, start + n))
        row_seq += [i] * n
        first.append(first[-1] + n)
    t = lambda v: torch.tensor(v, dtype=torch.int32, device=device)
    tiles = sorted(((i, r0) for i, s in enumerate(seqs) for r0 in range(0, s[2], 64)), key=lambda x: -x[1])
    tc = [x for x in tiles if x[1] % 128 == 0]
    tiles.sort(key=lambda x: -(seqs[x[0]][1] + x[1]))
    return SimpleNamespace(n_q_tiles=len(tiles) if any(s[2] > 1 for s in seqs) else 0,
                           n_q_tiles_tc=len(tc), q_tile_tc_seq=t([x[0] for x in tc]), q_tile_tc_row0=t([x[1] for x in tc]),
                           q_tile_seq=t([x[0] for x in tiles]), q_tile_row0=t([x[1] for x in tiles]),
                           row_pos=t(row_pos), row_seq=t(row_seq), seq_slot=t([s[0] for s in seqs]),
                           seq_first_row=t(first), seq_len=t([s[1] + s[2] for s in seqs]),
                           n_rows=len(row_pos), n_seqs=len(seqs), prefill=all(s[1] == 0 for s in seqs),
                           max_len=max(s[1] + s[2] for s in seqs), max_rows=max(s[2] for s in seqs))


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("nh,nkv,hd,rot", [(6, 2, 48, 48), (7, 7, 16, 16), (4, 1, 128, 64), (2, 2, 256, 256)])
def test_rope_append(K, dtype, nh, nkv, hd, rot):
    page = 16
    seqs = [(2, 0, 21), (0, 37, 1), (3, 5, 9)]
    tables = {2: [4, 1], 0: [7, 3, 9], 3: [0]}
    cpu, gpu = make_kv(10, nkv, page, hd, 4, 3, 0, 0, DT[dtype], tables)
    T = sum(s[2] for s in seqs)
    qkv = g(T, (nh + 2 * nkv) * hd, dtype=DT[dtype], seed=hd)
    inv = torch.pow(torch.tensor(12345.0, dtype=torch.float64), -2.0 * torch.arange(rot // 2, dtype=torch.float64) / rot).float()
    bc, bg = batch_of(seqs, "cpu"), batch_of(seqs, "cuda")
    want = qkv.clone()
    REF.rope_append(want, inv, rot, bc.row_pos, bc.row_seq, bc.seq_slot, bc.seq_len, cpu, nh, nkv, hd)
    got = qkv.cuda()
    K.rope_append(got, inv.cuda(), rot, bg.row_pos, bg.row_seq, bg.seq_slot, bg.seq_len, gpu, nh, nkv, hd)
    assert err(got, want) <= TOL[dtype]
    assert err(gpu.storage, cpu.storage) <= TOL[dtype]
    # pages of no sequence keep their stale contents
    for p in (2, 5, 6, 8):
        assert torch.all(gpu.storage[p].float() == 50.0)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_rope_append_long_prompt_wraps_a_ring(K, dtype):
    """A prompt longer than a windowed group's ring: every place must end up with its newest
    position, whichever block of the launch ran last."""
    nh, nkv, hd, page, window = 2, 2, 32, 16, 20
    ring = -(-window // page) + 1                      # 3 pages = 48 positions
    seqs = [(1, 0, 200), (0, 0, 30), (2, 0, 49)]
    tables = {1: [5, 0, 7], 0: [3, 8, 1], 2: [2, 4, 6]}
    cpu, gpu = make_kv(9, nkv, page, hd, 3, ring, ring, window, DT[dtype], tables)
    T = sum(s[2] for s in seqs)
    qkv = g(T, (nh + 2 * nkv) * hd, dtype=DT[dtype], seed=11)
    inv = torch.pow(torch.tensor(10000.0, dtype=torch.float64), -2.0 * torch.arange(hd // 2, dtype=torch.float64) / hd).float()
    bc, bg = batch_of(seqs, "cpu"), batch_of(seqs, "cuda")
    want = qkv.clone()
    REF.rope_append(want, inv, hd, bc.row_pos, bc.row_seq, bc.seq_slot, bc.seq_len, cpu, nh, nkv, hd)
    for _ in range(3):
        got = qkv.cuda()
        gpu.storage.fill_(50.0)
        K.rope_append(got, inv.cuda(), hd, bg.row_pos, bg.row_seq, bg.seq_slot, bg.seq_len, gpu, nh, nkv, hd)
        assert err(gpu.storage, cpu.storage) <= TOL[dtype]
    # position 199 of the long prompt is where the ring says, holding the rotated key of row 199
    e, off = (199 // page) % ring, 199 % page
    assert err(gpu.storage[tables[1][e], 0, :, off], want[199].view(-1, hd)[nh:nh + nkv]) <= TOL[dtype]


def test_rope_is_a_rotation_by_position_times_frequency(K):
    """Independent check: pair (i, i + d/2) as a complex number is multiplied by exp(i * p * f_i)."""
    nh, nkv, hd, theta = 2, 1, 32, 10000.0
    T = 5
    qkv = g(T, (nh + 2 * nkv) * hd, seed=1)
    pos = torch.tensor([0, 1, 17, 255, 4000], dtype=torch.int32)
    inv = torch.pow(torch.tensor(theta, dtype=torch.float64), -2.0 * torch.arange(hd // 2, dtype=torch.float64) / hd)
    got = qkv.cuda()
    z = torch.zeros(T, dtype=torch.int32, device="cuda")
    K.rope_append(got, inv.float().cuda(), hd, pos.cuda(), z, z[:1], z[:1], None, nh, nkv, hd)
    u = qkv.double().view(T, nh + 2 * nkv, hd)[:, :nh + nkv]
    c = torch.complex(u[..., :hd // 2], u[..., hd // 2:]) * torch.polar(torch.ones(T, hd // 2, dtype=torch.float64),
                                                                        pos.double()[:, None] * inv[None])[:, None, :]
    want = torch.cat([c.real, c.imag], dim=-1)
    gotq = got.cpu().double().view(T, nh + 2 * nkv, hd)
    assert (gotq[:, :nh + nkv] - want).abs().max().item() <= 3e-3 * 1e-2 + 4000 * 1.2e-7 * 4   # angle rounding at p = 4000
    assert torch.equal(gotq[:, nh + nkv:], qkv.double().view(T, -1, hd)[:, nh + nkv:])           # v untouched


def fill_cache(cpu, gpu, slot, k, v):
    """Write keys/values [n, nkv, hd] of positions 0..n-1 into a slot's pages (ring aware)."""
    for j in range(k.shape[0]):
        e = j // cpu.page_size
        if cpu.ring_pages:
            e %= cpu.ring_pages
        page = int(cpu.block_table[slot, e])
        cpu.storage[page, 0, :, j % cpu.page_size] = k[j]
        cpu.storage[page, 1, :, j % cpu.page_size] = v[j]
    gpu.storage.copy_(cpu.storage)


def scattered_tables(lens, slots, page, ring=0, seed=0):
    """Pages for each slot, drawn from a shuffled pool; returns (tables, pool size, table width)."""
    need = [min(-(-n // page), ring) if ring else -(-n // page) for n in lens]
    total = sum(need) + 3
    order = np.random.default_rng(seed).permutation(total).tolist()
    tables, k = {}, 0
    for slot, n in zip(slots, need):
        tables[slot] = order[k:k + n]
        k += n
    return tables, total, max(need)


@pytest.mark.parametrize("nh,nkv,hd", [(28, 4, 128), (14, 2, 64)])
def test_attention_decode_with_many_live_splits(K, nh, nkv, hd):
    """One sequence of 5,000 positions (79 pages) beside a short one: 33, 40 and 64 splits that all have pages (the
    short sequence's blocks beyond its pages have none), and the number the wrapper chooses for one long sequence
    alone (64), against the float64 statement; key 4,321 stands out for head 0."""
    lens, slots, page = [5000, 70], [2, 0], 64
    tables, n_pages, width = scattered_tables(lens, slots, page, seed=hd + 1)
    cpu, gpu = make_kv(n_pages, nkv, page, hd, 4, width, 0, 0, torch.bfloat16, tables)
    scale = 1.0 / math.sqrt(hd)
    qkv = g(2, (nh + 2 * nkv) * hd, dtype=torch.bfloat16, seed=5)
    for i, (slot, n) in enumerate(zip(slots, lens)):
        k, v = g(n, nkv, hd, dtype=torch.bfloat16, seed=30 + i), g(n, nkv, hd, dtype=torch.bfloat16, seed=40 + i)
        if i == 0:
            k[4321, 0] = qkv[0, :hd] * 6.0
        fill_cache(cpu, gpu, slot, k, v)
    seqs = [(slots[i], lens[i] - 1, 1) for i in range(2)]
    bc, bg = batch_of(seqs, "cpu"), batch_of(seqs, "cuda")
    want = torch.zeros(2, nh * hd, dtype=torch.float64)
    REF.attention_plain(qkv, cpu, bc.row_pos, bc.row_seq, bc.seq_slot, bc.seq_first_row, want, nh, nkv, hd, scale, 0, True)
    out = torch.empty(2, nh * hd, dtype=torch.bfloat16, device="cuda")
    for n_splits in (33, 40, 64):
        out.fill_(7.0)
        K.attention_decode(qkv.cuda(), gpu, bg.seq_slot, bg.seq_len, out, nh, nkv, hd, scale, 0, n_splits=n_splits)
        assert err(out, want) <= TOL["bfloat16"], n_splits
    from cima_b200.engine.profile import StepProfile
    K.profile = seen = StepProfile()
    try:
        out.fill_(7.0)
        K.attention_decode(qkv[:1].cuda(), gpu, bg.seq_slot[:1], bg.seq_len[:1], out[:1], nh, nkv, hd, scale, 0, max_len=5000)
    finally:
        K.profile = None
    assert [l.name for l in seen.launches] == ["attention_decode[64 splits]"]
    assert err(out[:1], want[:1]) <= TOL["bfloat16"]


@pytest.mark.parametrize("nh,nkv,hd,window,keep", [(14, 2, 64, 0, 0), (4, 4, 128, 40, 0), (6, 2, 48, 33, 5), (3, 1, 200, 64, 40), (40, 1, 64, 0, 0), (2, 1, 30, 96, 32)])
def test_attention_float32_the_same_bits_however_cut(K, nh, nkv, hd, window, keep):
    """A float32 row's attention from the step's own rows, from the cache with many rows at once and from the cache row by row: the
    same bits, around the borders of the 32-position pieces; with a sink, distance slopes and an infinity among the values that no
    earlier row may notice.  Against the float64 statement on the rows in front of that infinity."""
    n, page = 131, 16
    tables, n_pages, width = scattered_tables([n], [1], page, seed=hd)
    cpu, gpu = make_kv(n_pages, nkv, page, hd, 4, width, 0, 0, torch.float32, tables)
    qkv = g(n, (nh + 2 * nkv) * hd, seed=7)
    qkv[n - 1, (nh + nkv) * hd] = float("inf")
    fill_cache(cpu, gpu, 1, qkv[:, nh * hd:(nh + nkv) * hd].reshape(n, nkv, hd), qkv[:, (nh + nkv) * hd:].reshape(n, nkv, hd))
    scale, slopes = 1.0 / math.sqrt(hd), torch.linspace(0.0, 0.5, nh)
    more = dict(sink=1.0, keep_first=keep)
    bg, bc = batch_of([(1, 0, n)], "cuda"), batch_of([(1, 0, n)], "cpu")
    step, cached, alone = (torch.empty(n, nh * hd, device="cuda") for _ in range(3))
    args = (bg.row_pos, bg.row_seq, bg.seq_slot, bg.seq_first_row)
    K.attention_plain(qkv.cuda(), None, *args, step, nh, nkv, hd, scale, window, False, slopes=slopes.cuda(), **more)
    K.attention_plain(qkv.cuda(), gpu, *args, cached, nh, nkv, hd, scale, window, True, slopes=slopes.cuda(), **more)
    for i in range(n):
        b1 = batch_of([(1, i, 1)], "cuda")
        K.attention_plain(qkv[i:i + 1].cuda(), gpu, b1.row_pos, b1.row_seq, b1.seq_slot, b1.seq_first_row, alone[i:i + 1], nh, nkv, hd, scale,
                          window, True, slopes=slopes.cuda(), **more)
    assert torch.equal(step[:n - 1], cached[:n - 1]) and torch.equal(step[:n - 1], alone[:n - 1]) and bool(step[:n - 1].isfinite().all())
    want = torch.zeros(n, nh * hd, dtype=torch.float64)
    REF.attention_plain(qkv, None, bc.row_pos, bc.row_seq, bc.seq_slot, bc.seq_first_row, want, nh, nkv, hd, scale, window, False, slopes=slopes, **more)
    assert err(step[:n - 1], want[:n - 1]) <= TOL["float32"]


@pytest.mark.parametrize("nh,nkv,hd,window,keep", [(14, 2, 64, 0, 0), (6, 6, 64, 0, 0), (40, 2, 32, 50, 9), (12, 1, 96, 0, 0), (3, 3, 200, 64, 40), (2, 1, 30, 0, 0)])
def test_attention_float32_the_same_bits_in_any_company(K, nh, nkv, hd, window, keep):
    """Prompts of 1 to 131 rows and of 20 rows sixteen times in one step, and one more row of each from the cache in one step: each
    sequence as when it comes alone, whatever rows, teams and warps a block has there and whether the longest length is known."""
    page, rows = 16, [1, 5, 31, 32, 33, 64, 131] + [20] * 16
    n = len(rows)
    tables, n_pages, width = scattered_tables([r + 1 for r in rows], list(range(n)), page, seed=hd)
    cpu, gpu = make_kv(n_pages, nkv, page, hd, n, width, 0, 0, torch.float32, tables)
    qkv, last = g(sum(rows), (nh + 2 * nkv) * hd, seed=7), g(n, (nh + 2 * nkv) * hd, seed=8)
    first = [sum(rows[:i]) for i in range(n + 1)]
    for i, r in enumerate(rows):
        all_rows = torch.cat([qkv[first[i]:first[i] + r], last[i:i + 1]])
        fill_cache(cpu, gpu, i, all_rows[:, nh * hd:(nh + nkv) * hd].reshape(r + 1, nkv, hd), all_rows[:, (nh + nkv) * hd:].reshape(r + 1, nkv, hd))

    def run(seqs, x, cached, max_len):
        b, out = batch_of(seqs, "cuda"), torch.full((len(x), nh * hd), 7.0, device="cuda")
        K.attention_plain(x.cuda(), gpu if cached else None, b.row_pos, b.row_seq, b.seq_slot, b.seq_first_row, out, nh, nkv, hd, 1.0 / math.sqrt(hd), window,
                          cached, keep_first=keep, max_len=max_len)
        return out

    prompts = [(i, 0, r) for i, r in enumerate(rows)]
    whole, known = run(prompts, qkv, False, 0), run(prompts, qkv, False, max(rows))
    more = [(i, r, 1) for i, r in enumerate(rows)]
    steps, steps_known = run(more, last, True, 0), run(more, last, True, max(rows) + 1)
    assert torch.equal(whole, known) and torch.equal(steps, steps_known)
    for i, r in enumerate(rows[:9]):
        x = qkv[first[i]:first[i] + r]
        assert torch.equal(run([(i, 0, r)], x, False, r), whole[first[i]:first[i] + r]), r
        assert torch.equal(run([(i, 0, r)], x, True, 0), whole[first[i]:first[i] + r]), r
        assert torch.equal(run([(i, r, 1)], last[i:i + 1], True, r + 1)[0], steps[i]) and torch.equal(run([(i, r, 1)], last[i:i + 1], True, 0)[0], steps[i]), r
    bc, want = batch_of(prompts, "cpu"), torch.zeros(sum(rows), nh * hd, dtype=torch.float64)
    REF.attention_plain(qkv, None, bc.row_pos, bc.row_seq, bc.seq_slot, bc.seq_first_row, want, nh, nkv, hd, 1.0 / math.sqrt(hd), window, False, keep_first=keep)
    assert err(whole, want) <= TOL["float32"]


@pytest.mark.parametrize("dtype,hd,n_splits", [("float32", 64, 0), ("float32", 300, 0), ("bfloat16", 64, 1), ("bfloat16", 64, 3)])
def test_attention_without_a_sink_at_low_scores(K, dtype, hd, n_splits):
    """An ordinary softmax whose scores all lie near -150, from one key (a sequence's first row) to 140: the exponential of minus the
    maximum is infinite, and no entry is there for it to multiply.  ``n_splits``: the decode attention with so many splits (0: the plain
    kernels, the two head sizes on the two of them)."""
    nh, nkv, page, lens = 4, 2, 64, [1, 2, 65, 140]
    tables, n_pages, width = scattered_tables(lens, list(range(4)), page, seed=hd)
    cpu, gpu = make_kv(n_pages, nkv, page, hd, 4, width, 0, 0, DT[dtype], tables)
    scale, size = 1.0 / math.sqrt(hd), math.sqrt(150 / math.sqrt(hd))
    qkv = torch.full((4, (nh + 2 * nkv) * hd), -size).to(DT[dtype])
    for slot, n in enumerate(lens):
        fill_cache(cpu, gpu, slot, (size + 0.01 * g(n, nkv, hd, seed=slot)).to(DT[dtype]), g(n, nkv, hd, dtype=DT[dtype], seed=9 + slot))
    seqs = [(slot, n - 1, 1) for slot, n in enumerate(lens)]
    bc, bg = batch_of(seqs, "cpu"), batch_of(seqs, "cuda")
    want = torch.zeros(4, nh * hd, dtype=torch.float64)
    REF.attention_plain(qkv, cpu, bc.row_pos, bc.row_seq, bc.seq_slot, bc.seq_first_row, want, nh, nkv, hd, scale, 0, True)
    out = torch.full((4, nh * hd), 7.0, dtype=DT[dtype], device="cuda")
    if n_splits:
        K.attention_decode(qkv.cuda(), gpu, bg.seq_slot, bg.seq_len, out, nh, nkv, hd, scale, 0, n_splits=n_splits)
    else:
        K.attention_plain(qkv.cuda(), gpu, bg.row_pos, bg.row_seq, bg.seq_slot, bg.seq_first_row, out, nh, nkv, hd, scale, 0, True)
    # float32: a score of 150 is off by the sum's steps, hd half ulps of it at most, and its exponential by that factor
    assert err(out, want) <= (TOL["bfloat16"] if dtype == "bfloat16" else 2 * hd * 150 * 2.0 ** -24 * want.abs().max().item())


@pytest.mark.parametrize("dtype,page", [("float32", 16), ("bfloat16", 16), ("bfloat16", 64)])
@pytest.mark.parametrize("nh,nkv,hd", [(6, 2, 48), (7, 1, 128), (4, 4, 16), (28, 4, 128), (3, 3, 80), (40, 2, 64), (2, 1, 112)])
def test_attention_decode_over_cache(K, dtype, page, nh, nkv, hd):
    """Three sequences of unequal length in scattered pages; a far key stands out in one of them.
    Pages of 64 in bfloat16 take the split-KV tensor-core kernel, the others the plain one."""
    lens = [300, 1, 77]
    slots = [1, 3, 0]
    tables, n_pages, width = scattered_tables(lens, slots, page, seed=hd)
    cpu, gpu = make_kv(n_pages, nkv, page, hd, 4, width, 0, 0, DT[dtype], tables)
    scale = 1.0 / math.sqrt(hd)
    qkv = g(3, (nh + 2 * nkv) * hd, dtype=DT[dtype], seed=3)
    for i, (slot, n) in enumerate(zip(slots, lens)):
        k, v = g(n, nkv, hd, dtype=DT[dtype], seed=10 + i), g(n, nkv, hd, dtype=DT[dtype], seed=20 + i)
        if i == 0:
            # key 13 of 300 is the query of head 0 scaled up: nearly all the weight falls on it
            k[13, 0] = qkv[0, :hd] * 6.0
        fill_cache(cpu, gpu, slot, k, v)
    seqs = [(slots[i], lens[i] - 1, 1) for i in range(3)]
    bc, bg = batch_of(seqs, "cpu"), batch_of(seqs, "cuda")
    want = torch.zeros(3, nh * hd, dtype=torch.float64)
    REF.attention_plain(qkv, cpu, bc.row_pos, bc.row_seq, bc.seq_slot, bc.seq_first_row, want, nh, nkv, hd, scale, 0, True)
    out = torch.empty(3, nh * hd, dtype=DT[dtype], device="cuda")
    K.attention(qkv.cuda(), gpu, bg, out, nh, nkv, hd, scale, 0, True)
    assert err(out, want) <= TOL[dtype]
    plain = torch.empty_like(out)
    K.attention_plain(qkv.cuda(), gpu, bg.row_pos, bg.row_seq, bg.seq_slot, bg.seq_first_row, plain, nh, nkv, hd, scale, 0, True)
    assert err(plain, want) <= TOL[dtype]
    if dtype == "bfloat16" and page == 64:
        # more splits than pages too; up to 8 merge inside a cluster, more through a second kernel; ``early``
        # fetches the first pages before the wait on the previous kernel (which here writes ``out`` only)
        for n_splits in (1, 2, 3, 5, 8, 9, 32):
            for early in (False, True):
                out.fill_(7.0)
                K.attention_decode(qkv.cuda(), gpu, bg.seq_slot, bg.seq_len, out, nh, nkv, hd, scale, 0,
                                   n_splits=n_splits, early=early)
                assert err(out, want) <= TOL[dtype], (n_splits, early)


@pytest.mark.parametrize("dtype,page", [("float32", 16), ("bfloat16", 16), ("bfloat16", 64)])
@pytest.mark.parametrize("window,n", [(40, 200), (16, 17), (33, 33), (64, 500), (100, 1000), (1, 70)])
def test_attention_decode_window_edge(K, dtype, page, window, n):
    """A ring of pages; the key just outside the window stands out and must not be seen, the one just
    inside must."""
    nh, nkv, hd = 4, 2, 32
    ring = -(-window // page) + 1
    tables, n_pages, width = scattered_tables([n], [1], page, ring=ring, seed=window)
    cpu, gpu = make_kv(n_pages, nkv, page, hd, 2, ring, ring, window, DT[dtype], tables)
    scale = 1.0 / math.sqrt(hd)
    qkv = g(1, (nh + 2 * nkv) * hd, dtype=DT[dtype], seed=4)
    k, v = g(n, nkv, hd, dtype=DT[dtype], seed=5), g(n, nkv, hd, dtype=DT[dtype], seed=6)
    inside, outside = n - window, n - window - 1
    if outside >= 0:
        k[outside, 0] = qkv[0, :hd] * 8.0          # would take all the weight of head 0 if it were seen
    k[inside, 1] = qkv[0, 2 * hd:3 * hd] * 8.0     # head 2 reads kv head 1: must be seen
    # only what a ring still holds: the newest positions
    fill_cache(cpu, gpu, 1, k, v)
    bg = batch_of([(1, n - 1, 1)], "cuda")
    # the statement: plain softmax over the visible keys of the full, unwrapped sequence
    want = torch.zeros(1, nh * hd, dtype=torch.float64)
    for h in range(nh):
        gk = h // (nh // nkv)
        lo = max(0, n - window)
        s = (k[lo:n, gk].double() @ qkv[0, h * hd:(h + 1) * hd].double()) * scale
        want[0, h * hd:(h + 1) * hd] = torch.softmax(s, 0) @ v[lo:n, gk].double()
    out = torch.empty(1, nh * hd, dtype=DT[dtype], device="cuda")
    K.attention(qkv.cuda(), gpu, bg, out, nh, nkv, hd, scale, window, True)
    assert err(out, want) <= TOL[dtype]
    assert err(out[0, 2 * hd:3 * hd], v[inside, 1]) <= 5e-2      # head 2 is (nearly) that one value
    if dtype == "bfloat16" and page == 64:
        for n_splits in (1, 2, 7, 8, 16):
            for early in (False, True):
                out.fill_(7.0)
                K.attention_decode(qkv.cuda(), gpu, bg.seq_slot, bg.seq_len, out, nh, nkv, hd, scale, window,
                                   n_splits=n_splits, early=early)
                assert err(out, want) <= TOL[dtype], (n_splits, early)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("nh,nkv,hd,window", [(6, 2, 48, 0), (7, 1, 128, 0), (4, 2, 64, 50), (2, 2, 256, 0),
                                              (28, 4, 128, 0), (5, 5, 16, 7), (4, 2, 96, 64), (2, 1, 32, 65),
                                              (3, 1, 112, 200), (2, 2, 80, 1)])
def test_attention_prefill_over_the_step(K, dtype, nh, nkv, hd, window):
    """Ragged prompts in one launch; keys and values come from the step's own rows."""
    lens = [130, 1, 67, 300]
    seqs = [(i, 0, n) for i, n in enumerate(lens)]
    T = sum(lens)
    scale = 1.0 / math.sqrt(hd)
    qkv = g(T, (nh + 2 * nkv) * hd, dtype=DT[dtype], seed=hd + nh)
    # in the last sequence, key 5 stands out for the last query of head 0 (a far key among hundreds)
    last = T - 1
    first4 = T - 300
    qkv[first4 + 5, nh * hd:(nh + 1) * hd] = qkv[last, :hd] * 6.0
    bc, bg = batch_of(seqs, "cpu"), batch_of(seqs, "cuda")
    want = torch.zeros(T, nh * hd, dtype=torch.float64)
    REF.attention_plain(qkv, None, bc.row_pos, bc.row_seq, bc.seq_slot, bc.seq_first_row, want, nh, nkv, hd, scale, window, False)
    out = torch.empty(T, nh * hd, dtype=DT[dtype], device="cuda")
    K.attention(qkv.cuda(), None, bg, out, nh, nkv, hd, scale, window, False)
    assert err(out, want) <= TOL[dtype]
    plain = torch.empty_like(out)
    K.attention_plain(qkv.cuda(), None, bg.row_pos, bg.row_seq, bg.seq_slot, bg.seq_first_row, plain, nh, nkv, hd, scale, window, False)
    assert err(plain, want) <= TOL[dtype]


@pytest.mark.parametrize("lens", [[130, 1, 67, 300], [128], [1], [257, 256, 255], [700, 40]])
@pytest.mark.parametrize("nh,nkv,window", [(7, 1, 0), (4, 2, 0), (28, 4, 0), (4, 2, 50), (2, 2, 200), (3, 1, 128), (2, 1, 1)])
@pytest.mark.parametrize("hd", [128, 64])
def test_attention_prefill_tcgen05(K, lens, nh, nkv, window, hd):
    """The tcgen05 attention of ragged prompts (head_dim 64 and 128) against the float64 statement: sequences that
    end inside a block of 128, a far key that stands out, windows with edges inside and between tiles."""
    seqs = [(i, 0, n) for i, n in enumerate(lens)]
    T = sum(lens)
    scale = 1.0 / math.sqrt(hd)
    qkv = g(T, (nh + 2 * nkv) * hd, dtype=torch.bfloat16, seed=nh + T)
    if lens[-1] > 6 and (window == 0 or window >= lens[-1]):
        # in the last sequence, key 5 stands out for the last query of head 0 (a far key among hundreds)
        qkv[T - lens[-1] + 5, nh * hd:(nh + 1) * hd] = qkv[T - 1, :hd] * 6.0
    bc, bg = batch_of(seqs, "cpu"), batch_of(seqs, "cuda")
    want = torch.zeros(T, nh * hd, dtype=torch.float64)
    REF.attention_plain(qkv, None, bc.row_pos, bc.row_seq, bc.seq_slot, bc.seq_first_row, want, nh, nkv, hd, scale, window, False)
    out = torch.full((T, nh * hd), 7.0, dtype=torch.bfloat16, device="cuda")
    K.attention_prefill_tc(qkv.cuda(), bg, out, nh, nkv, hd, scale, window)
    assert K.device_errors() == 0
    assert err(out, want) <= TOL["bfloat16"]


def first_launch_on_long_sequences(n_seqs=8, n=8192, nh=28, nkv=4, hd=128):
    """Run by the test below in a process of its own, where the launch is the kernel's first: then its loads are
    slow (nothing of the buffer is in any cache or translation buffer) and the roles of a block drift apart."""
    from cima_b200.kernels import Kernels
    K = Kernels(verbose=False)
    T = n_seqs * n
    gen = torch.Generator(device="cuda").manual_seed(3)
    qkv = torch.randn(T, (nh + 2 * nkv) * hd, generator=gen, device="cuda", dtype=torch.float32).to(torch.bfloat16)
    bg = batch_of([(i, 0, n) for i in range(n_seqs)], "cuda")
    out = torch.full((T, nh * hd), 7.0, dtype=torch.bfloat16, device="cuda")
    scale = 1.0 / math.sqrt(hd)
    K.attention_prefill_tc(qkv, bg, out, nh, nkv, hd, scale, 0)
    assert K.device_errors() == 0, "a bounded wait ran out in the kernel's first launch"
    for seq, h in ((0, 0), (n_seqs - 1, nh - 1), (n_seqs // 2, nh // 2)):     # some heads whole, in float64
        rows = slice(seq * n, (seq + 1) * n)
        kvh = h // (nh // nkv)
        q = qkv[rows, h * hd:(h + 1) * hd].double()
        k = qkv[rows, (nh + kvh) * hd:(nh + kvh + 1) * hd].double()
        v = qkv[rows, (nh + nkv + kvh) * hd:(nh + nkv + kvh + 1) * hd].double()
        sc = (q @ k.T) * scale
        sc.masked_fill_(torch.ones(n, n, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
        want = torch.softmax(sc, dim=-1) @ v
        got = out[rows, h * hd:(h + 1) * hd].double()
        assert (got - want).abs().max().item() <= TOL["bfloat16"], (seq, h)
    print("first launch sound")


def test_attention_prefill_tcgen05_long_sequences_of_64_wide_heads():
    """Four sequences of 8,192 rows with 14 heads of 64 in 2 groups (128 key tiles a block at the narrow head size),
    three heads whole against float64."""
    first_launch_on_long_sequences(n_seqs=4, n=8192, nh=14, nkv=2, hd=64)


@pytest.mark.parametrize("attempt", [0, 1])
def test_attention_prefill_tcgen05_first_launch_on_long_sequences(attempt):
    """Eight sequences of 8,192 rows at the 7B head shape as the first launch of a fresh process.  With one barrier for
    the probabilities of both score buffers, the softmax warps could announce two tiles while the issuing thread
    still waited for a late tile of V, and its wait was answered a phase late: about every second fresh process ran
    into the bounded wait.  Two processes, since the drift is a matter of timing."""
    import os, subprocess, sys
    here = os.path.dirname(os.path.abspath(__file__))
    code = f"import sys; sys.path[:0] = [{here!r}, {os.path.dirname(here)!r}]; import test_kernels_gpu as t; t.first_launch_on_long_sequences()"
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "first launch sound" in r.stdout, r.stdout[-2000:] + r.stderr[-2000:]


@pytest.mark.parametrize("nh,nkv,hd", [(6, 2, 48), (28, 4, 128), (4, 4, 16)])
@pytest.mark.parametrize("window,ring", [(0, 0), (90, 0), (40, 2)])
def test_attention_of_sequences_that_go_on(K, nh, nkv, hd, window, ring):
    """Several query rows per sequence over the paged cache (the step's own keys are in the pages too) against the
    float64 statement: a sequence deep into its cache, one that starts, one across a page's edge, one with more than
    two blocks of rows; stale keys behind every sequence's end; a window, and a window through a ring of two pages."""
    page = 64
    seqs = [(2, 100, 64), (0, 0, 5), (3, 63, 2)] + ([] if ring else [(1, 500, 150)])
    width = ring or 11
    order = torch.randperm(4 * width, generator=torch.Generator().manual_seed(5)).tolist()
    tables = {slot: order[slot * width:(slot + 1) * width] for slot in range(4)}
    cpu, gpu = make_kv(4 * width, nkv, page, hd, 4, width, ring, window, torch.bfloat16, tables)
    cpu.storage.copy_(g(*cpu.storage.shape, dtype=torch.bfloat16, seed=hd + window))
    gpu.storage.copy_(cpu.storage)
    T = sum(s[2] for s in seqs)
    scale = 1.0 / math.sqrt(hd)
    qkv = g(T, (nh + 2 * nkv) * hd, dtype=torch.bfloat16, seed=nh + T)
    bc, bg = batch_of(seqs, "cpu"), batch_of(seqs, "cuda")
    want = torch.zeros(T, nh * hd, dtype=torch.float64)
    REF.attention_plain(qkv, cpu, bc.row_pos, bc.row_seq, bc.seq_slot, bc.seq_first_row, want, nh, nkv, hd, scale, window, True)
    out = torch.full((T, nh * hd), 7.0, dtype=torch.bfloat16, device="cuda")
    K.attention_extend(qkv.cuda(), gpu, bg, out, nh, nkv, hd, scale, window)
    assert err(out, want) <= TOL["bfloat16"]
    # the dispatcher takes the same kernel for such a batch
    out2 = torch.full((T, nh * hd), 7.0, dtype=torch.bfloat16, device="cuda")
    K.attention(qkv.cuda(), gpu, bg, out2, nh, nkv, hd, scale, window, True)
    assert torch.equal(out, out2)


@pytest.mark.parametrize("nh,nkv,hd", [(12, 2, 128), (6, 2, 48), (3, 1, 16)])
@pytest.mark.parametrize("window,keep", [(0, 0), (300, 0), (130, 70)])
def test_attention_of_going_on_rows_with_shared_keys(K, nh, nkv, hd, window, keep):
    """The key tiles of a block of rows shared by 2, 5 and 64 blocks (more than there are tiles: some have none), for a sequence
    deep into its cache, one that starts and one whose rows cross a page's edge; with a sink, a stored number a head, distance slopes
    and gates; against the float64 statement and the launch that is not split."""
    seqs, page, width = [(2, 1900, 70), (0, 0, 5), (1, 126, 3)], 64, 31
    order = torch.randperm(4 * width, generator=torch.Generator().manual_seed(7)).tolist()
    tables = {slot: order[slot * width:(slot + 1) * width] for slot in range(4)}
    cpu, gpu = make_kv(4 * width, nkv, page, hd, 4, width, 0, window, torch.bfloat16, tables)
    cpu.storage.copy_(g(*cpu.storage.shape, dtype=torch.bfloat16, seed=hd + window))
    gpu.storage.copy_(cpu.storage)
    T, scale, cols = sum(s[2] for s in seqs), 1.0 / math.sqrt(hd), (nh + 2 * nkv) * hd
    qkv = g(T, cols + nh * hd, dtype=torch.bfloat16, seed=nh + T)
    bc, bg = batch_of(seqs, "cpu"), batch_of(seqs, "cuda")
    slopes, head_sink = torch.linspace(0.0, 0.02, nh), torch.linspace(-1.0, 2.0, nh)
    for kw in (dict(sink=1.0), dict(head_sink=head_sink, slopes=slopes), dict(gate_col=cols)):
        want = torch.zeros(T, nh * hd, dtype=torch.float64)
        REF.attention_plain(qkv, cpu, bc.row_pos, bc.row_seq, bc.seq_slot, bc.seq_first_row, want, nh, nkv, hd, scale, window, True, keep_first=keep, **kw)
        dev = {k: v.cuda() if torch.is_tensor(v) else v for k, v in kw.items()}
        whole = torch.full((T, nh * hd), 7.0, dtype=torch.bfloat16, device="cuda")
        K.attention_extend(qkv.cuda(), gpu, bg, whole, nh, nkv, hd, scale, window, keep_first=keep, n_splits=1, **dev)
        assert err(whole, want) <= TOL["bfloat16"]
        for n_splits in (2, 5, 64):
            out = torch.full((T, nh * hd), 7.0, dtype=torch.bfloat16, device="cuda")
            K.attention_extend(qkv.cuda(), gpu, bg, out, nh, nkv, hd, scale, window, keep_first=keep, n_splits=n_splits, **dev)
            assert err(out, want) <= TOL["bfloat16"], (n_splits, list(kw))


@pytest.mark.parametrize("nh,nkv,hd,v_group", [(8, 4, 64, 2), (4, 2, 128, 1), (4, 4, 128, 4)])
@pytest.mark.parametrize("window,keep", [(90, 70), (300, 5), (64, 200), (130, 64), (0, 0)])
def test_attention_tcgen05_with_kept_positions_and_shared_values(K, nh, nkv, hd, v_group, window, keep):
    """The tcgen05 attention where a window keeps first positions (none of them below it, some, whole tiles, more than the window's
    first rows have) and key heads share value heads: prompts on their own rows, and sequences that go on from the cache; the
    dispatcher takes it for both."""
    nv, page, width, scale = nkv // v_group, 64, 9, 1.0 / math.sqrt(hd)
    for seqs, cached in ([(0, 0, 420), (1, 0, 37)], False), ([(2, 100, 260), (0, 0, 5), (1, 380, 130)], True):
        T, cols = sum(s[2] for s in seqs), (nh + nkv + nv) * hd
        qkv = g(T, cols, dtype=torch.bfloat16, seed=nh + T)
        bc, bg = batch_of(seqs, "cpu"), batch_of(seqs, "cuda")
        cpu = gpu = None
        if cached:
            order = torch.randperm(4 * width, generator=torch.Generator().manual_seed(6)).tolist()
            cpu, gpu = make_kv(4 * width, nkv, page, hd, 4, width, 0, window, torch.bfloat16, {s: order[s * width:(s + 1) * width] for s in range(4)})
            cpu.storage.copy_(g(*cpu.storage.shape, dtype=torch.bfloat16, seed=hd + window + 1))
            gpu.storage.copy_(cpu.storage)
        want = torch.zeros(T, nh * hd, dtype=torch.float64)
        REF.attention_plain(qkv, cpu, bc.row_pos, bc.row_seq, bc.seq_slot, bc.seq_first_row, want, nh, nkv, hd, scale, window, cached, keep_first=keep, v_group=v_group)
        out = torch.full((T, nh * hd), 7.0, dtype=torch.bfloat16, device="cuda")
        K.attention_prefill_tc(qkv.cuda(), bg, out, nh, nkv, hd, scale, window, kv=gpu, keep_first=keep, v_group=v_group)
        assert K.device_errors() == 0
        assert err(out, want) <= TOL["bfloat16"], cached
        out2 = torch.full((T, nh * hd), 7.0, dtype=torch.bfloat16, device="cuda")
        K.attention(qkv.cuda(), gpu, bg, out2, nh, nkv, hd, scale, window, cached, keep_first=keep, v_group=v_group)
        assert torch.equal(out, out2), cached


@pytest.mark.parametrize("spread", [1.0, 2.0])
@pytest.mark.parametrize("T,nh,nkv,hd,v_group,window,keep", [(700, 24, 4, 64, 2, 0, 0), (1100, 16, 4, 64, 2, 512, 64), (900, 12, 2, 128, 1, 300, 64)])
def test_attention_tcgen05_as_near_to_64_bits_as_mma_sync(K, T, nh, nkv, hd, v_group, window, keep, spread):
    """The forms that came to the tcgen05 kernel from the mma.sync one, from flat scores to rows of a few large probabilities: prompts
    and the same rows from the cache.  Both round each probability to bfloat16 once, the largest being exactly 1, and here the denominator
    has the same roundings: no further off than there."""
    nv, scale = nkv // v_group, 1.0 / math.sqrt(hd)
    qkv = g(T, (nh + nkv + nv) * hd, dtype=torch.bfloat16, seed=T, scale=spread).cuda()
    b = batch_of([(0, 0, T)], "cuda")
    q, k, v = (t.double().view(T, -1, hd).transpose(0, 1) for t in qkv.split([nh * hd, nkv * hd, nv * hd], dim=1))
    i = torch.arange(T, device="cuda")
    seen = i[None] <= i[:, None]
    if window:
        seen &= (i[:, None] - i[None] < window) | (i[None] < keep)
    want = torch.stack([(q[h] @ k[h // (nh // nkv)].t() * scale).masked_fill(~seen, -math.inf).softmax(-1) @ v[h // (nh // nkv) // v_group] for h in range(nh)], 1).reshape(T, -1)
    pages = -(-T // 64)
    cpu, gpu = make_kv(pages, nkv, 64, hd, 1, pages, 0, window, torch.bfloat16, {0: list(range(pages))})
    fill_cache(cpu, gpu, 0, qkv[:, nh * hd:(nh + nkv) * hd].view(T, nkv, hd).cpu(), torch.nn.functional.pad(qkv[:, (nh + nkv) * hd:].view(T, nv, hd), (0, 0, 0, nkv - nv)).cpu())
    off = {}
    for name, call in (("mma", lambda o: K.attention_prefill(qkv, b.q_tile_seq, b.q_tile_row0, b.seq_first_row, o, nh, nkv, hd, scale, window, keep_first=keep, v_group=v_group)),
                       ("tc", lambda o: K.attention_prefill_tc(qkv, b, o, nh, nkv, hd, scale, window, keep_first=keep, v_group=v_group)),
                       ("tc cached", lambda o: K.attention_prefill_tc(qkv, b, o, nh, nkv, hd, scale, window, kv=gpu, keep_first=keep, v_group=v_group))):
        o = torch.empty(T, nh * hd, dtype=torch.bfloat16, device="cuda")
        call(o)
        off[name] = ((o.double() - want).norm() / want.norm()).item()
    assert K.device_errors() == 0
    assert max(off["tc"], off["tc cached"]) <= off["mma"], off


@pytest.mark.parametrize("nh,nkv,hd", [(4, 2, 128), (6, 1, 64)])
@pytest.mark.parametrize("window", [0, 90, 300])
def test_attention_of_sequences_that_go_on_by_many_rows_tcgen05(K, nh, nkv, hd, window):
    """The tcgen05 attention with its keys from the cache's pages (by TMA through the block table): a sequence of 260
    rows deep into its cache, one that starts, one of 130 rows; stale keys behind every end; windows."""
    page = 64
    seqs = [(2, 100, 260), (0, 0, 5), (1, 380, 130)]
    width = 9
    order = torch.randperm(4 * width, generator=torch.Generator().manual_seed(6)).tolist()
    tables = {slot: order[slot * width:(slot + 1) * width] for slot in range(4)}
    cpu, gpu = make_kv(4 * width, nkv, page, hd, 4, width, 0, window, torch.bfloat16, tables)
    cpu.storage.copy_(g(*cpu.storage.shape, dtype=torch.bfloat16, seed=hd + window + 1))
    gpu.storage.copy_(cpu.storage)
    T = sum(s[2] for s in seqs)
    scale = 1.0 / math.sqrt(hd)
    qkv = g(T, (nh + 2 * nkv) * hd, dtype=torch.bfloat16, seed=nh + T)
    bc, bg = batch_of(seqs, "cpu"), batch_of(seqs, "cuda")
    want = torch.zeros(T, nh * hd, dtype=torch.float64)
    REF.attention_plain(qkv, cpu, bc.row_pos, bc.row_seq, bc.seq_slot, bc.seq_first_row, want, nh, nkv, hd, scale, window, True)
    out = torch.full((T, nh * hd), 7.0, dtype=torch.bfloat16, device="cuda")
    K.attention_prefill_tc(qkv.cuda(), bg, out, nh, nkv, hd, scale, window, kv=gpu)
    assert K.device_errors() == 0
    assert err(out, want) <= TOL["bfloat16"]
    out2 = torch.full((T, nh * hd), 7.0, dtype=torch.bfloat16, device="cuda")
    K.attention(qkv.cuda(), gpu, bg, out2, nh, nkv, hd, scale, window, True)      # the dispatcher's choice for such a batch
    assert torch.equal(out, out2)


# ---------------------------------------------------------------------------- sampling
def test_argmax_ties_go_to_the_higher_index(K):
    V = 1000
    x = g(5, V, seed=1)
    x[0, 17] = x[0, 900] = 9.0
    x[1, :] = -3.0
    x[2, 999] = 50.0
    x[3, 0] = 50.0
    tok = torch.empty(5, dtype=torch.int32, device="cuda")
    K.argmax(x.cuda(), tok)
    assert tok.tolist() == [900, 999, 999, 0, int(torch.nonzero(x[4] == x[4].max()).max())]


# ---------------------------------------------------------------------------- norm folded into the skinny product
@pytest.mark.parametrize("M", [1, 5, 7, 8])
@pytest.mark.parametrize("N,K_", [(200, 328), (4608, 3584), (1000, 192)])
def test_skinny_accumulate_leaves_sums_of_squares_and_the_next_product_folds_the_norm(K, M, N, K_):
    """x += a W1^T leaves per-tile sums of squares of the updated rows; the next product takes the rows,
    the norm's weight and those sums and must equal RMSNorm followed by the product."""
    from cima_b200.kernels import SK_ACCUM, SK_STORE, SK_STORE_F32, SK_SWIGLU
    H = K_
    a = g(M, N, dtype=torch.bfloat16, seed=1)
    w1 = g(H, N, dtype=torch.bfloat16, seed=2, scale=1.0 / math.sqrt(N))
    x0 = g(M, H, seed=3)
    x = x0.cuda()
    ssq = torch.full((M, -(-H // 16)), -1.0, device="cuda")
    K.linear_skinny(a.cuda(), w1.cuda(), None, x, SK_ACCUM, ssq)
    want_x = x0.double() + a.double() @ w1.double().t()
    assert err(x, want_x) <= 1e-4
    assert err(ssq.sum(dim=1), (x.double() ** 2).sum(dim=1)) <= 1e-3 * max(1.0, float((want_x ** 2).sum(dim=1).max()))
    # the writer also leaves the rows times the next norm's weight; the product after the norm reads those
    nw = 1 + g(H, seed=4, scale=0.1)
    xb = x0.cuda()
    ssq_b = torch.full_like(ssq, -1.0)
    xw = torch.full((M, H), 9.0, dtype=torch.bfloat16, device="cuda")
    K.linear_skinny(a.cuda(), w1.cuda(), None, xb, SK_ACCUM, ssq_b, nw.cuda(), xw)
    assert torch.equal(xb, x) and torch.equal(ssq_b, ssq)
    assert torch.equal(xw, (x * nw.cuda()).to(torch.bfloat16))
    eps = 1e-5
    xd = x.double().cpu()
    h = (xd / torch.sqrt((xd * xd).mean(dim=1, keepdim=True) + eps) * nw.double())
    w2 = g(2 * 96, H, dtype=torch.bfloat16, seed=5, scale=1.0 / math.sqrt(H))
    b2 = g(2 * 96, seed=6)
    want = h @ w2.double().t()
    out = torch.empty(M, 192, dtype=torch.bfloat16, device="cuda")
    K.linear_skinny_norm(xw, ssq, eps, w2.cuda(), b2.cuda(), out, SK_STORE)
    assert err(out, want + b2.double()) <= TOL["bfloat16"] * 4
    out32 = torch.empty(M, 192, device="cuda")
    K.linear_skinny_norm(xw, ssq, eps, w2.cuda(), None, out32, SK_STORE_F32)
    # the operand is bf16(x * w): one bfloat16 rounding per term against the float64 statement
    assert err(out32, want) <= TOL["bfloat16"] * 2
    act = torch.empty(M, 96, dtype=torch.bfloat16, device="cuda")
    K.linear_skinny_norm(xw, ssq, eps, w2.cuda(), None, act, SK_SWIGLU)
    gg, uu = want[:, :96], want[:, 96:]
    assert err(act, gg / (1 + torch.exp(-gg)) * uu) <= TOL["bfloat16"] * 4


def test_embed_leaves_sums_of_squares(K):
    table = g(300, 200, dtype=torch.bfloat16)
    ids = torch.tensor([0, 299, 7], dtype=torch.int32)
    x = torch.empty(3, 200, device="cuda")
    ssq = torch.empty(3, 1, device="cuda")
    K.embed(ids.cuda(), table.cuda(), x, 1.0, ssq)
    assert err(ssq[:, 0], (table[ids.long()].double() ** 2).sum(dim=1)) <= 1e-3
    nw = (1 + g(200, seed=4, scale=0.1)).cuda()
    x2, ssq2 = torch.empty_like(x), torch.empty_like(ssq)
    xw = torch.empty(3, 200, dtype=torch.bfloat16, device="cuda")
    K.embed(ids.cuda(), table.cuda(), x2, 1.0, ssq2, nw, xw)
    assert torch.equal(x2, x) and torch.equal(ssq2, ssq)
    assert torch.equal(xw, (x * nw).to(torch.bfloat16))


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("T,H", [(5, 200), (64, 3584), (300, 1000)])
def test_add_rmsnorm_equals_the_two_kernels(K, dtype, T, H):
    x0, d, w = g(T, H, seed=1, scale=2.0), g(T, H, dtype=DT[dtype], seed=2), 1 + g(H, seed=3, scale=0.1)
    xa, xb = x0.cuda(), x0.cuda()
    ha = torch.empty(T, H, dtype=DT[dtype], device="cuda")
    hb = torch.empty_like(ha)
    K.add_rmsnorm(xa, d.cuda(), w.cuda(), 1e-5, ha)
    K.add_residual(xb, d.cuda())
    K.rmsnorm(xb, w.cuda(), 1e-5, hb)
    assert torch.equal(xa, xb) and torch.equal(ha, hb)
    want = torch.empty(T, H, dtype=torch.float64)
    REF.rmsnorm(x0 + d.float(), w, 1e-5, want)
    assert err(ha, want) <= TOL[dtype] * 4


@pytest.mark.parametrize("M,N,K_", [(256, 256, 64), (300, 328, 200), (2048, 1000, 448), (513, 3584, 192), (130, 66, 72),
                                    (1, 8, 8), (257, 264, 72), (1000, 200, 136)])
def test_gemm_tcgen05_pair_modes(K, M, N, K_):
    """The product on pairs of SMs (cta_group::2) against float64, every epilogue, tails in every dimension (a last
    tile of rows that starts early to end with the matrix must store, and above all accumulate, its own rows only)."""
    from cima_b200.kernels import SK_ACCUM, SK_STORE, SK_STORE_F32, SK_SWIGLU
    a = g(M, K_, dtype=torch.bfloat16, seed=M)
    w = g(N, K_, dtype=torch.bfloat16, seed=N, scale=1.0 / math.sqrt(K_))
    b = g(N, seed=7)
    want = a.double() @ w.double().t()
    out32 = torch.full((M, N), -777.0, device="cuda")
    K.gemm_tc_pair(a.cuda(), w.cuda(), b.cuda(), out32, SK_STORE_F32)
    assert err(out32, want + b.double()) <= 1e-4
    out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    K.gemm_tc_pair(a.cuda(), w.cuda(), None, out, SK_STORE)
    assert err(out, want) <= TOL["bfloat16"] * 4
    x = g(M, N, seed=9)
    xg = x.cuda()
    K.gemm_tc_pair(a.cuda(), w.cuda(), None, xg, SK_ACCUM)
    assert err(xg, x.double() + want) <= 1e-4
    if N % 2 == 0:
        I = N // 2
        gg, uu = want[:, :I], want[:, I:]
        for code in (0, 1, 2, 3):                       # the gate's activation: SiLU, GELU (tanh, erf), ReLU
            act = torch.empty(M, I, dtype=torch.bfloat16, device="cuda")
            K.gemm_tc_pair(a.cuda(), w.cuda(), None, act, SK_SWIGLU, act=code)
            assert err(act, REF.gate_act(gg, code) * uu) <= TOL["bfloat16"] * 4, code
    assert K.device_errors() == 0


def test_gemm_tcgen05_pair_gate_over_its_whole_range(K):
    """SiLU in the gated epilogue, gates of either sign from 1e-30 to 1e30 and every hundredth up to 130: float32's quotient and
    exponential (2 ulp) in front of the rounding to bfloat16 (8 bits: at most 2^-8 of the value).  The exponential of a gate below -88.72 is
    infinite, so less than 89 * 2^-128 goes there, times the up value's 3 at most; down to it nothing does, so an infinite up value
    stays infinite."""
    from cima_b200.kernels import SK_SWIGLU
    v = torch.cat([torch.arange(-13000, 13000).double() / 100, 10.0 ** torch.arange(-30, 31).double(), -10.0 ** torch.arange(-30, 31).double(), torch.zeros(1).double()])
    v = v.to(torch.bfloat16)
    a, w = torch.zeros(len(v), 8, dtype=torch.bfloat16), torch.zeros(32, 8, dtype=torch.bfloat16)
    a[:, 0], a[:, 1] = v, 1.0
    w[:16, 0], w[16:, 1] = 1.0, torch.linspace(-3, 3, 16).to(torch.bfloat16)
    out = torch.empty(len(v), 16, dtype=torch.bfloat16, device="cuda")
    K.gemm_tc_pair(a.cuda(), w.cuda(), None, out, SK_SWIGLU)
    want = (v.double() * torch.sigmoid(v.double()))[:, None] * w[16:, 1].double()
    assert bool(((out.cpu().double() - want).abs() <= 2.0 ** -8 * (1 + 2.0 ** -12) * want.abs() + 89 * 2.0 ** -128 * 3).all())
    w[16:, 1] = float("inf")
    K.gemm_tc_pair(a.cuda(), w.cuda(), None, out, SK_SWIGLU)
    some = (v > -88.7) & (v != 0)
    assert torch.equal(out.cpu()[some].float(), (torch.sign(v[some].float()) * float("inf"))[:, None].expand(-1, 16))
    assert K.device_errors() == 0


@pytest.mark.parametrize("inter,width,rows,fused", [(40, 768, 943, False), (40, 768, 1500, False), (72, 1536, 236, False), (72, 1536, 300, False),
                                                    (40, 3072, 251, False), (24, 760, 1024, False), (40, 3072, 256, True), (40, 3072, 501, False),
                                                    (40, 3072, 502, True), (24, 3064, 512, False),
                                                    (24, 1536, 1024, True), (24, 1528, 1024, False), (24, 1536, 1023, False), (24, 1536, 1254, False),
                                                    (24, 1536, 1255, True)])
def test_gated_pair_on_the_kernel_its_rule_picks(K, inter, width, rows, fused):
    """Rows and sums on both sides of the rule that picks the fused tcgen05 product or the library's and the activation kernel, and
    which of them ran.  Tolerance: gate, up and their product rounded to bfloat16 each, 2^-8 of the largest value they can pass on."""
    from cima_b200.engine.profile import StepProfile
    from cima_b200.parts.linear import GatedLinearPair
    from cima_b200.parts.runtime import Runtime
    gate, up = (g(inter, width, dtype=torch.bfloat16, seed=s, scale=1.0 / math.sqrt(width)) for s in (1, 2))
    pair = GatedLinearPair(gate, up, Runtime(kernels=K, dtype=torch.bfloat16, device="cuda:0"))
    a = g(rows, width, dtype=torch.bfloat16, seed=rows)
    K.profile = seen = StepProfile()
    try:
        got = pair.activated(a.cuda())
    finally:
        K.profile = None
    names = [launch.name for launch in seen.launches]
    assert any("tcgen05" in n for n in names) == fused and any("swiglu" in n for n in names) != fused, names
    z = a.double() @ pair.lin.weight.cpu().double().t()
    want = REF.gate_act(z[:, :inter], 0) * z[:, inter:]
    assert err(got, want) <= 3 * 2.0 ** -8 * (z[:, :inter].abs().max() * z[:, inter:].abs().max()).item()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("nh,nkv,hd,rotary,nd", [(5, 2, 64, 64, 64), (28, 4, 128, 64, 128), (3, 1, 16, 0, 8)])
def test_norm_rotation_and_append_the_same_bits_for_any_number_of_rows(K, nh, nkv, hd, rotary, nd, dtype):
    """Rows that a launch gives a warp one, two and four heads of (few, hundreds, 2,048 and more), at the lines between: each row and
    its keys and values in the pages as when it comes alone; against the float64 statement."""
    heads, T = nh + 2 * nkv, 2100
    edge = 1800 // -(-heads // 4)
    qkv = g(T, heads * hd, dtype=DT[dtype], seed=hd)
    inv, norm = torch.rand(rotary // 2, generator=torch.Generator().manual_seed(2)), [1 + g(nd, seed=s, scale=0.1) for s in (3, 4)]
    pages = -(-T // 64)

    def run(first, n):
        cpu, gpu = make_kv(pages, nkv, 64, hd, 1, pages, 0, 0, DT[dtype], {0: list(range(pages))})
        b = batch_of([(0, first, n)], "cuda")
        q = qkv[first:first + n].contiguous().cuda()
        K.rope_append(q, inv.cuda(), rotary, b.row_pos, b.row_seq, b.seq_slot, torch.tensor([first + n], dtype=torch.int32, device="cuda"), gpu, nh, nkv, hd,
                      qk_norm=(norm[0].cuda(), norm[1].cuda(), nd, 1e-6))
        return q, gpu.storage.transpose(2, 3).reshape(pages, 2, 64, nkv, hd).transpose(1, 2).reshape(pages * 64, 2, nkv, hd)[first:first + n]

    whole, kept = run(0, T)
    for n in (edge, edge + 1, 2047, 2048):
        part, kept_part = run(0, n)
        assert torch.equal(part, whole[:n]) and torch.equal(kept_part, kept[:n]), n
    for first in (0, 1, 777, T - 1):
        part, kept_part = run(first, 1)
        assert torch.equal(part[0], whole[first]) and torch.equal(kept_part[0], kept[first]), first
    x = qkv.double().view(T, heads, hd)[:, :nh + nkv].clone()
    r = 1.0 / torch.sqrt((x[..., :nd] ** 2).mean(-1, keepdim=True) + 1e-6)
    w = torch.cat([norm[0].double().expand(nh, nd), norm[1].double().expand(nkv, nd)])
    x[..., :nd] = x[..., :nd] * r * w
    if rotary:
        # the angle as the kernel has it, a float32 product: its sine and cosine move by that rounding, not by the kernel's own
        angle = (torch.arange(T).float()[:, None] * inv).double()[:, None]
        a, c = x[..., :rotary // 2].clone(), x[..., rotary // 2:rotary].clone()
        x[..., :rotary // 2], x[..., rotary // 2:rotary] = a * angle.cos() - c * angle.sin(), a * angle.sin() + c * angle.cos()
    assert err(whole[:, :(nh + nkv) * hd], x.reshape(T, -1)) <= TOL[dtype] * x.abs().max().item()
    assert torch.equal(whole[:, nh * hd:].view(T, 2, nkv, hd)[:, 0], kept[:, 0]) and torch.equal(whole[:, nh * hd:].view(T, 2, nkv, hd)[:, 1], kept[:, 1])


@pytest.mark.parametrize("M", [1, 5, 7, 8])
@pytest.mark.parametrize("nh,nkv,hd,H", [(6, 2, 48, 200), (28, 4, 128, 3584), (3, 1, 64, 192), (4, 4, 16, 64)])
def test_qkv_rope_skinny_equals_projection_then_rope_append(K, M, nh, nkv, hd, H):
    """The decode projection with rotation and cache append in its epilogue against the two separate steps
    (float64 statement): rotated q in the buffer, rotated k and v in the right pages, other pages untouched."""
    from cima_b200.kernels import SK_ACCUM
    page = 64
    N = (nh + 2 * nkv) * hd
    lens = [int(x) for x in np.random.default_rng(M).integers(1, 200, size=M)]
    slots = list(np.random.default_rng(M + 1).permutation(M + 3)[:M])
    tables, n_pages, width = scattered_tables(lens, slots, page, seed=hd + M)
    cpu, gpu = make_kv(n_pages, nkv, page, hd, M + 3, width, 0, 0, torch.bfloat16, tables)
    seqs = [(int(slots[i]), lens[i] - 1, 1) for i in range(M)]
    bc, bg = batch_of(seqs, "cpu"), batch_of(seqs, "cuda")
    a = g(M, H, dtype=torch.bfloat16, seed=1)
    w = g(N, H, dtype=torch.bfloat16, seed=2, scale=1.0 / math.sqrt(H))
    b = g(N, seed=3, scale=0.5)
    inv = torch.pow(torch.tensor(10000.0, dtype=torch.float64), -2.0 * torch.arange(hd // 2, dtype=torch.float64) / hd).float()
    # statement: projection in float64, rotation and append by the reference (rounded once at the end)
    want = (a.double() @ w.double().t() + b.double())
    REF.rope_append(want, inv, hd, bc.row_pos, bc.row_seq, bc.seq_slot, bc.seq_len, cpu, nh, nkv, hd)
    qkv = torch.full((M, N), 7.0, dtype=torch.bfloat16, device="cuda")
    K.qkv_rope(a.cuda(), w.cuda(), b.cuda(), qkv, inv.cuda(), bg.row_pos, bg.row_seq, bg.seq_slot, gpu, nh, nkv, hd)
    assert err(qkv[:, :nh * hd], want[:, :nh * hd]) <= TOL["bfloat16"] * 4
    assert err(gpu.storage, cpu.storage) <= TOL["bfloat16"] * 4
    # with the norm folded in: rows times the norm's weight and partial sums of squares, as an accumulating
    # product leaves them
    x = g(M, H, seed=4, scale=1.5).cuda()
    nw = (1 + g(H, seed=5, scale=0.1))
    ssq = torch.empty(M, -(-H // 16), device="cuda")
    xw = torch.empty(M, H, dtype=torch.bfloat16, device="cuda")
    zero_w = torch.zeros(H, 8, dtype=torch.bfloat16, device="cuda")
    K.linear_skinny(torch.zeros(M, 8, dtype=torch.bfloat16, device="cuda"), zero_w, None, x, SK_ACCUM, ssq, nw.cuda(), xw)
    xd = x.double().cpu()
    hh = xd / torch.sqrt((xd * xd).mean(dim=1, keepdim=True) + 1e-6) * nw.double()
    want2 = hh @ w.double().t() + b.double()
    cpu2, gpu2 = make_kv(n_pages, nkv, page, hd, M + 3, width, 0, 0, torch.bfloat16, tables)
    REF.rope_append(want2, inv, hd, bc.row_pos, bc.row_seq, bc.seq_slot, bc.seq_len, cpu2, nh, nkv, hd)
    K.qkv_rope(xw, w.cuda(), b.cuda(), qkv, inv.cuda(), bg.row_pos, bg.row_seq, bg.seq_slot, gpu2, nh, nkv, hd,
               norm=(ssq, 1e-6))
    assert err(qkv[:, :nh * hd], want2[:, :nh * hd]) <= TOL["bfloat16"] * 4
    assert err(gpu2.storage, cpu2.storage) <= TOL["bfloat16"] * 4


@pytest.mark.parametrize("nh,nkv,hd,window", [(14, 2, 64, 0), (15, 3, 64, 40), (16, 2, 128, 0), (28, 4, 128, 129)])
def test_float32_attention_of_few_rows_has_the_bits_of_many(K, nh, nkv, hd, window):
    """Decode rows in 32 bits, one head a block while they are few, and together with others, as many rows share a block's keys: the
    same bits at the ends of a piece (32 positions), a page (64) and a block's round (256), and near float64."""
    lens = [1, 2, 31, 32, 33, 63, 64, 65, 128, 255, 256, 257, 300, 513, 700]
    lens += lens[:max(0, 296 // nh + 1 - len(lens))]
    B = len(lens)
    assert B * nh > 296
    tables, n_pages, width = scattered_tables(lens, list(range(B)), 64, seed=hd + window)
    cpu, gpu = make_kv(n_pages, nkv, 64, hd, B, width, 0, window, torch.float32, tables)
    cpu.storage.fill_(float("nan"))                       # what no row sees is not read
    for i, n in enumerate(lens):
        fill_cache(cpu, gpu, i, g(n, nkv, hd, seed=50 + i), g(n, nkv, hd, seed=90 + i))
    qkv, scale = g(B, (nh + 2 * nkv) * hd, seed=6), 1.0 / math.sqrt(hd)
    seqs = [(i, n - 1, 1) for i, n in enumerate(lens)]

    def run(which):
        b = batch_of([seqs[i] for i in which], "cuda")
        out = torch.full((len(which), nh * hd), 7.0, device="cuda")
        K.attention_plain(qkv[which].cuda(), gpu, b.row_pos, b.row_seq, b.seq_slot, b.seq_first_row, out, nh, nkv, hd, scale, window, True)
        return out

    many = run(list(range(B)))
    for i in range(B):
        assert torch.equal(run([i])[0], many[i]), lens[i]
    assert torch.equal(run([0, B - 1, 3]), many[[0, B - 1, 3]])
    bc, want = batch_of(seqs, "cpu"), torch.zeros(B, nh * hd, dtype=torch.float64)
    REF.attention_plain(qkv, cpu, bc.row_pos, bc.row_seq, bc.seq_slot, bc.seq_first_row, want, nh, nkv, hd, scale, window, True)
    assert err(many, want) <= TOL["float32"]


@pytest.mark.parametrize("nh,nkv,hd,window", [(6, 2, 64, 40), (4, 1, 64, 129), (2, 2, 128, 64), (12, 2, 128, 200)])
def test_float32_attention_of_few_rows_over_a_ring(K, nh, nkv, hd, window):
    """A window's keys in a ring of pages that has wrapped several times: pieces of 32 keys whose lower part newer positions have
    overwritten.  Against float64 over the whole sequences; the key just below the window stands out until it is left out."""
    lens, ring, scale = [1, window - 1, window, window + 1, 449, 640, 707, 1025], -(-window // 64) + 1, 1.0 / math.sqrt(hd)
    B, G = len(lens), nh // nkv
    assert B * nh <= 296
    slots = list(range(B))
    tables = {i: [ring * i + j for j in range(ring)] for i in slots}
    cpu, gpu = make_kv(ring * B, nkv, 64, hd, B, ring, ring, window, torch.float32, tables)
    qkv = g(B, (nh + 2 * nkv) * hd, seed=6)
    want = torch.empty(B, nh * hd, dtype=torch.float64)
    for i, n in enumerate(lens):
        k, v, lo = g(n, nkv, hd, seed=50 + i), g(n, nkv, hd, seed=90 + i), max(0, n - window)
        if lo:
            k[lo - 1, 0] = 9.0 * qkv[i, :hd]
        fill_cache(cpu, gpu, i, k, v)
        for h in range(nh):
            p = torch.softmax((k[lo:, h // G].double() @ qkv[i, h * hd:(h + 1) * hd].double()) * scale, 0)
            want[i, h * hd:(h + 1) * hd] = p @ v[lo:, h // G].double()
    b, out = batch_of([(i, n - 1, 1) for i, n in enumerate(lens)], "cuda"), torch.full((B, nh * hd), 7.0, device="cuda")
    K.attention_plain(qkv.cuda(), gpu, b.row_pos, b.row_seq, b.seq_slot, b.seq_first_row, out, nh, nkv, hd, scale, window, True)
    assert err(out, want) <= TOL["float32"]
