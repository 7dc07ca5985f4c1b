"""The decode attention whose blocks are clusters that merge their own results: every cluster size at the edges of its pieces (16 keys a
warp, 128 a block, pages of 64), windows and rings against float64; and which step takes it."""
import math
from types import SimpleNamespace

import pytest
import torch

from cima_b200.cache.kv import LayerKV
from cima_b200.kernels import Kernels, decode_splits, near_cluster, near_context

TOL = 2e-2          # bfloat16 values of magnitude 1 to 4 and their weighted means, as in test_kernels_gpu.py
LENS = [1, 2, 16, 17, 64, 65, 128, 129, 300, 1100]


def test_the_rule_covers_every_number_of_pairs():
    """At most one block an SM (two at head size 64) where a cluster has more than one."""
    for hd, room in ((64, 296), (128, 148)):
        last = 16
        for pairs in range(1, 600):
            c = near_cluster(pairs, hd)
            assert c in (1, 2, 4, 8, 16) and c <= last and (c == 1 or pairs * c <= room)
            last = c


ROOM = {64: (14, 33, 71, 148), 128: (7, 15, 33, 74)}              # what a B200 answered
# (head size, pairs, positions): us a layer of the cluster kernel against the splits, sequences of one length, on a B200
FASTER = {(128, 4, 8000): -3.0, (128, 8, 4000): -3.2, (128, 12, 8000): -2.3, (128, 14, 16000): -2.3, (128, 16, 2000): -3.6, (128, 20, 16000): -4.5,
          (128, 32, 16000): -3.5, (128, 33, 6000): -3.0, (128, 36, 700): -2.3, (128, 40, 700): -3.5, (128, 48, 2000): -1.3, (128, 56, 4000): -1.3,
          (128, 60, 12000): -4.7, (128, 74, 4000): -3.4, (128, 76, 700): -2.5, (128, 96, 700): -2.9, (128, 104, 8000): -9.4, (128, 128, 4000): -4.9,
          (128, 152, 4000): -3.7, (128, 256, 4000): -1.5, (64, 2, 8000): -0.9, (64, 24, 16000): -8.0, (64, 32, 2000): -1.7, (64, 56, 16000): -4.5,
          (64, 71, 2000): -3.1, (64, 96, 4000): -1.6, (64, 128, 4000): -7.6, (64, 176, 4000): -13.2}
SLOWER = {(128, 2, 16000): 0.4, (128, 16, 6000): 1.9, (128, 36, 6000): 7.3, (128, 38, 4000): 3.0, (128, 40, 4000): 1.6, (128, 48, 8000): 5.1, (128, 48, 16000): 14.0,
          (128, 56, 8000): 1.3, (128, 76, 4000): 4.6, (128, 92, 4000): 3.9, (128, 96, 4000): 3.5, (128, 96, 8000): 12.1, (64, 2, 16000): 0.4,
          (64, 16, 16000): 1.5, (64, 32, 16000): 2.6}


def test_the_reach_lies_where_it_was_measured():
    """No number of pairs at a length at which the splits were faster, and every one well below."""
    for (hd, pairs, n), us in {**FASTER, **SLOWER}.items():
        reach = near_context(pairs, 1, hd, ROOM[hd])
        assert (reach == 0 or n <= reach) == (us < 0), (hd, pairs, n, reach, near_cluster(pairs, hd, ROOM[hd]), decode_splits(pairs))


# (head size, sequences, kv heads, positions of one, the others having 300): the same
FASTER_UNEVEN = {(128, 16, 2, 2000): -1.5, (128, 3, 4, 8000): -4.2, (128, 6, 4, 30000): -15.7, (128, 8, 4, 30000): -15.8, (128, 32, 4, 700): -2.9, (128, 40, 4, 30000): -151.0,
                 (128, 64, 4, 1000): -8.8, (64, 8, 2, 4000): -0.6, (64, 24, 2, 4000): -1.1, (64, 64, 2, 30000): -34.4, (64, 48, 2, 2000): -0.6,
                 (128, 8, 8, 30000): -12.2, (128, 7, 8, 4000): -3.8, (128, 4, 8, 30000): -16.7, (64, 6, 8, 16000): -7.0, (64, 3, 8, 16000): -12.0}
SLOWER_UNEVEN = {(128, 6, 2, 8000): 0.9, (128, 7, 2, 16000): 4.1, (128, 10, 2, 4000): 0.1, (128, 16, 2, 8000): 2.1, (128, 22, 2, 2000): 1.4, (128, 28, 2, 4000): 3.8,
                 (128, 12, 4, 2000): 0.3, (128, 16, 4, 4000): 1.3, (128, 24, 4, 2000): 2.8, (128, 32, 4, 4000): 2.6, (128, 60, 2, 4000): 3.4, (64, 8, 2, 8000): 1.1,
                 (64, 16, 2, 4000): 0.2, (64, 24, 2, 8000): 0.4, (64, 48, 2, 4000): 0.4, (128, 5, 8, 4000): 2.0, (128, 7, 8, 30000): 7.3, (128, 9, 8, 4000): 1.3, (64, 9, 8, 2000): 1.0}


def test_the_reach_with_one_long_sequence_lies_where_it_was_measured():
    for (hd, n_seqs, nkv, n), us in {**FASTER_UNEVEN, **SLOWER_UNEVEN}.items():
        reach = near_context(n_seqs, nkv, hd, ROOM[hd], even=False)
        assert (reach == 0 or n <= reach) == (us < 0), (hd, n_seqs, nkv, n, reach)


def test_which_step_takes_it():
    """The dispatch itself: head sizes, groups, planes, alignment, unknown lengths, windows, short contexts, unevenness."""
    def near(nh=14, nkv=2, hd=64, rows=1, max_len=1000, window=0, planes=2, width=None, ptr=0, even=True):
        self = SimpleNamespace(near_room=ROOM.get)
        qkv = SimpleNamespace(shape=(rows, (nh + 2 * nkv) * hd if width is None else width), data_ptr=lambda: ptr)
        return Kernels._near(self, qkv, SimpleNamespace(planes=planes), SimpleNamespace(n_rows=rows, max_len=max_len, even=even), nh, nkv, hd, window)

    assert near() == 16 and near(nh=28, nkv=4, hd=128) == 16
    assert near(hd=96) == near(hd=256) == near(nh=18, nkv=2) == near(planes=1) == near(width=1004) == near(ptr=8) == 0
    assert near(max_len=384) == 1 and near(max_len=385) == 16 and near(hd=128, max_len=192) == 1
    assert near(max_len=832 * 16) == 16 and near(max_len=832 * 16 + 1) == 0 == near(max_len=0)
    assert near(nh=28, nkv=4, hd=128, rows=64, max_len=0) == 1                                     # as many blocks as splits: at any length
    assert near(nh=28, nkv=4, hd=128, rows=9, max_len=2000) == 0 and near(nh=28, nkv=4, hd=128, rows=9, max_len=1664) == 2
    assert near(max_len=10 ** 6, window=300) == 1 and near(max_len=0, window=1000) == 16 and near(max_len=10 ** 6, window=20000) == 0
    assert near(nh=28, nkv=4, hd=128, rows=32, max_len=4000) == 1 and near(nh=28, nkv=4, hd=128, rows=32, max_len=4000, even=False) == 0
    assert near(nh=28, nkv=4, hd=128, rows=32, max_len=900, even=False) == 1 and near(nh=28, nkv=4, hd=128, rows=8, max_len=30000, even=False) == 4


def test_the_clusters_are_those_that_the_device_holds():
    """A device whose groups of SMs hold fewer clusters, or none of a size: never more blocks to wait for one another than it can place."""
    for hd in (64, 128):
        for room in ((0, 0, 0, 0), (0, 14, 33, 72), (2, 6, 12, 30), (0, 0, 35, 74), (100, 100, 100, 200)):
            for pairs in range(1, 200):
                c = near_cluster(pairs, hd, room)
                assert c == 1 or pairs <= room[{16: 0, 8: 1, 4: 2, 2: 3}[c]]


@pytest.mark.gpu
@pytest.mark.parametrize("nh,nkv,hd,window,more", [
    (14, 2, 64, 0, ""), (28, 4, 128, 0, "early"), (6, 6, 128, 0, ""), (8, 1, 64, 0, "early"), (6, 2, 128, 40, "early"), (4, 4, 64, 129, "ring"),
    (15, 3, 64, 64, "ring early")])
def test_attention_near(nh, nkv, hd, window, more):
    K, B, page, G = Kernels(verbose=False), len(LENS), 64, nh // nkv
    gen = torch.Generator().manual_seed(nh + hd + window)
    randn = lambda *s: torch.randn(*s, generator=gen)                                           # noqa: E731
    ring = -(-window // page) + 1 if "ring" in more else 0
    width = ring or -(-max(LENS) // page)
    storage = torch.full((B * width + 3, 2, nkv, page, hd), float("nan"), dtype=torch.bfloat16)      # what no sequence holds must not be seen
    table = torch.randperm(B * width + 3, generator=gen)[:B * width].view(B, width).int()
    slots = torch.randperm(B, generator=gen).int()
    qkv = randn(B, (nh + 2 * nkv) * hd).bfloat16()
    want = torch.empty(B, nh * hd, dtype=torch.float64)
    for b, n in enumerate(LENS):
        k, v = randn(n, nkv, hd).bfloat16(), randn(n, nkv, hd).bfloat16()
        lo = max(0, n - window) if window else 0
        k[lo, 0] = qkv[b, :hd] * 3.0                               # the oldest visible key stands out for head 0, the one below it more
        if lo:
            k[lo - 1, 0] = qkv[b, :hd] * 9.0
        for p in range(max(0, n - ring * page + page) if ring else 0, n):
            e = (p // page) % ring if ring else p // page
            at = table[slots[b], e]
            storage[at, 0, :, p % page], storage[at, 1, :, p % page] = k[p], v[p]
        for h in range(nh):
            s = (k[lo:, h // G].double() @ qkv[b, h * hd:(h + 1) * hd].double()) * 0.3 / math.sqrt(hd)
            want[b, h * hd:(h + 1) * hd] = torch.softmax(s, 0) @ v[lo:, h // G].double()
    kv = LayerKV(storage.cuda(), table.cuda(), page, ring, window, 0)
    args = (qkv.cuda(), kv, slots.cuda(), torch.tensor(LENS, dtype=torch.int32, device="cuda"))
    for cluster in (1, 2, 4, 8, 16):
        out = torch.full((B, nh * hd), 7.0, dtype=torch.bfloat16, device="cuda")
        K.attention_decode_near(*args, out, nh, nkv, hd, 0.3 / math.sqrt(hd), window, cluster, early="early" in more)
        got = out.cpu().double()
        assert ((got - want).abs() <= TOL * want.abs().clamp(min=1.0)).all(), (cluster, (got - want).abs().max().item())
    one = torch.full((1, nh * hd), 7.0, dtype=torch.bfloat16, device="cuda")      # a sequence alone: the same bits
    K.attention_decode_near(qkv[-1:].cuda(), kv, slots[-1:].cuda(), args[3][-1:], one, nh, nkv, hd, 0.3 / math.sqrt(hd), window, 16, early="early" in more)
    assert torch.equal(one[0], out[-1])


@pytest.mark.gpu
@pytest.mark.parametrize("hd", [64, 128])
def test_an_infinite_value_stays_in_its_column(hd):
    """130 positions: a warp's second 16 keys end after two, and what it has read before of the other fourteen must not come back."""
    K, n = Kernels(verbose=False), 130
    storage = torch.zeros(3, 2, 1, 64, hd, dtype=torch.bfloat16)
    storage[0, 1, 0, 5, 3] = float("inf")                          # weight 1 / 130
    kv = LayerKV(storage.cuda(), torch.arange(3, dtype=torch.int32, device="cuda").view(1, 3), 64, 0, 0, 0)
    out = torch.full((1, 2 * hd), 7.0, dtype=torch.bfloat16, device="cuda")
    slot, length = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.full((1,), n, dtype=torch.int32, device="cuda")
    K.attention_decode_near(torch.ones(1, 4 * hd, dtype=torch.bfloat16, device="cuda"), kv, slot, length, out, 2, 1, hd, 1.0, 0, 1)
    want = torch.zeros(2, hd, dtype=torch.bfloat16)
    want[:, 3] = float("inf")
    assert torch.equal(out.cpu().view(2, hd), want)


@pytest.mark.gpu
@pytest.mark.parametrize("nh,nkv,hd,B", [(28, 4, 128, 80), (14, 2, 64, 170)])
def test_more_blocks_than_one_wave(nh, nkv, hd, B):
    """Some hundred sequences of 1 to 700 positions, up to 5,440 blocks: every row against float64."""
    K, G, gen, width = Kernels(verbose=False), nh // nkv, torch.Generator().manual_seed(hd), 11
    lens = torch.randint(1, 700, (B,), generator=gen).int()
    storage = torch.randn(B * width, 2, nkv, 64, hd, generator=gen).bfloat16().cuda()
    table, slots = torch.randperm(B * width, generator=gen).view(B, width).int(), torch.randperm(B, generator=gen)
    qkv = torch.randn(B, (nh + 2 * nkv) * hd, generator=gen).bfloat16().cuda()
    held = storage[table[slots].long().cuda()].double().permute(0, 2, 3, 1, 4, 5).reshape(B, 2, nkv, width * 64, hd)
    seen = (torch.arange(width * 64) < lens[:, None]).cuda()
    s = (qkv[:, :nh * hd].double().view(B, nkv, G, hd) @ held[:, 0].transpose(2, 3) / math.sqrt(hd)).masked_fill(~seen[:, None, None], -math.inf)
    want = (torch.softmax(s, -1) @ held[:, 1]).reshape(B, nh * hd)
    kv = LayerKV(storage, table.cuda(), 64, 0, 0, 0)
    for cluster in (1, 2, 4, 8, 16):
        out = torch.full((B, nh * hd), 7.0, dtype=torch.bfloat16, device="cuda")
        K.attention_decode_near(qkv, kv, slots.int().cuda(), lens.cuda(), out, nh, nkv, hd, 1.0 / math.sqrt(hd), 0, cluster)
        assert ((out.double() - want).abs() <= TOL * want.abs().clamp(min=1.0)).all(), cluster


@pytest.mark.gpu
@pytest.mark.parametrize("signs", ["mixed", "one"])
@pytest.mark.parametrize("nh,nkv,hd", [(14, 2, 64), (28, 4, 128)])
def test_long_sums_are_as_near_to_64_bits_as_the_splits(nh, nkv, hd, signs):
    """Values of mixed and of one sign, up to 8,000 positions: no cluster is further from float64 than the split kernel at 64 splits, whose
    sums are the shortest (2 % for what the rounding of the result leaves to chance)."""
    K, B, G = Kernels(verbose=False), 4, nh // nkv
    for n in (300, 2000, 8000):
        gen, width = torch.Generator().manual_seed(n + hd), -(-n // 64)
        storage = torch.randn(B * width, 2, nkv, 64, hd, generator=gen)
        if signs == "one":
            storage[:, 1] = storage[:, 1].abs()
        storage = storage.bfloat16().cuda()
        table = torch.randperm(B * width, generator=gen).view(B, width).int().cuda()
        qkv = torch.randn(B, (nh + 2 * nkv) * hd, generator=gen).bfloat16().cuda()
        held = storage[table.long()].double().permute(0, 2, 3, 1, 4, 5).reshape(B, 2, nkv, width * 64, hd)[..., :n, :]
        q, scale = qkv[:, :nh * hd].double().view(B, nkv, G, hd), 1.0 / math.sqrt(hd)
        want = (torch.softmax(q @ held[:, 0].transpose(2, 3) * scale, -1) @ held[:, 1]).reshape(B, nh * hd)
        args = (qkv, LayerKV(storage, table, 64, 0, 0, 0), torch.arange(B, dtype=torch.int32, device="cuda"), torch.full((B,), n, dtype=torch.int32, device="cuda"))
        out = torch.empty(B, nh * hd, dtype=torch.bfloat16, device="cuda")
        off = lambda: ((out.double() - want).norm() / want.norm()).item()                          # noqa: E731
        K.attention_decode(*args, out, nh, nkv, hd, scale, 0, n_splits=64)
        splits = off()
        for cluster in (1, 2, 4, 8, 16):
            K.attention_decode_near(*args, out, nh, nkv, hd, scale, 0, cluster)
            assert off() <= 1.02 * splits, (n, cluster, off(), splits)


@pytest.mark.gpu
def test_clusters_stay_within_what_the_device_holds(monkeypatch):
    """The device is asked once, and a step takes no cluster that it cannot place: with room for none of 16 (as where no group has 16 free
    SMs) the step runs in smaller ones."""
    K = Kernels(verbose=False)
    for hd in (64, 128):
        room = K.near_room(hd)
        assert len(room) == 4 and room[3] > 0 and all(a <= b for a, b in zip(room, room[1:])), room
        assert K.near_room(hd) is room
        qkv, kv = torch.zeros(1, 4 * hd, dtype=torch.bfloat16, device="cuda"), SimpleNamespace(planes=2)
        batch = SimpleNamespace(n_rows=1, n_seqs=1, max_len=1000)
        assert K._near(qkv, kv, batch, 2, 1, hd, 0) == near_cluster(1, hd, room)
        K._near_room[(torch.cuda.current_device(), hd)] = (0,) + room[1:]
        assert K._near(qkv, kv, batch, 2, 1, hd, 0) == 8


@pytest.mark.gpu
def test_steps_cross_the_reach_of_the_clusters(monkeypatch):
    """Decoding across the bound behind which the splits take over (lowered, so that a short walk crosses it): the same logits as
    steps that are issued one by one, to the rounding of bfloat16."""
    import cima_b200
    from cima_b200 import kernels
    from cima_b200.config.shapes import SHAPES
    from cima_b200.engine import StepEntry
    monkeypatch.setattr(kernels, "NEAR_KEYS", 32)                   # 512 positions for a cluster of 16
    kw = dict(config=dict(SHAPES["qwen2.5-0.5b"], num_hidden_layers=2, max_position_embeddings=4096), seed=3, draw="device", max_tokens=4096, max_seqs=2, verbose=False)
    rec, ref, splits = cima_b200.load(**kw), cima_b200.load(use_graphs=False, **kw), cima_b200.load(use_graphs=False, **kw)
    splits.model.rt.kernels._near = lambda *a: 0                    # (another kernel altogether)
    prompt = torch.randint(0, rec.spec.vocab, (505,), generator=torch.Generator().manual_seed(1)).tolist()
    outs = []
    for lm in (rec, ref, splits):
        (slot,) = lm.model.cache.open(1)
        lm.step([StepEntry(slot, prompt)])
        outs.append(torch.cat([lm.step([StepEntry(slot, [t], [0])]) for t in range(100, 116)]))
    assert {k[1] for k in rec.model._step_graphs} == {512, 0}
    assert (outs[0] - outs[1]).abs().max() <= 2e-2 * outs[1].std()
    assert (outs[0] - outs[2]).abs().max() <= 2e-2 * outs[2].std()


@pytest.mark.gpu
@pytest.mark.parametrize("shape,seqs,longest,want", [("qwen2.5-0.5b", 25, 6137, {0, -1}), ("qwen2.5-1.5b", 10, 3836, {0, -1}), ("qwen2.5-7b", 3, 500, {0})])
def test_steps_of_sequences_far_from_one_length(shape, seqs, longest, want):
    """One long sequence beside short ones: its steps are recorded apart from where the splits are the faster ones for it, and the logits
    stay those of the split kernel, step by step (two layers; the clusters are of 4, 4 and 8 blocks)."""
    import cima_b200
    from cima_b200.config.shapes import SHAPES
    from cima_b200.engine import StepEntry
    from cima_b200.engine.graph import UNEVEN
    kw = dict(config=dict(SHAPES[shape], num_hidden_layers=2, max_position_embeddings=8192), seed=3, draw="device", max_tokens=16384, max_seqs=seqs, verbose=False)
    rec, ref = cima_b200.load(**kw), cima_b200.load(use_graphs=False, **kw)
    ref.model.rt.kernels._near = lambda *a: 0
    g, outs = torch.Generator().manual_seed(1), []
    prompts = [torch.randint(0, rec.spec.vocab, (longest if i == 0 else 20 + i,), generator=g).tolist() for i in range(seqs)]
    for lm in (rec, ref):
        slots = lm.model.cache.open(seqs)
        lm.step([StepEntry(s, p) for s, p in zip(slots, prompts)])
        outs.append([lm.step([StepEntry(s, [t + i], [0]) for i, s in enumerate(slots)]) for t in range(100, 114)])
    for n, (a, b) in enumerate(zip(*outs)):                       # each is up to 0.7 % off its 64-bit result
        assert ((a - b).norm(dim=1) <= 1.5e-2 * b.norm(dim=1)).all(), n
    assert UNEVEN == -1 and {k[1] for k in rec.model._step_graphs} == want


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [3, 11])
@pytest.mark.parametrize("nh,nkv,hd", [(14, 2, 64), (28, 4, 128)])
def test_the_newest_position_is_read_behind_its_append(rows, nh, nkv, hd, monkeypatch):
    """The kernel that rotates and appends (the skinny product's epilogue up to 8 rows, the rotation by itself above), then at once the
    attention by every cluster: NaN stands in the cache at the newest position until the append, whose key is the row's own query
    of head 0 and outweighs the others.  Against append and softmax in float64."""
    from reference_kernels import ReferenceKernels
    from test_kernels_gpu import batch_of, fill_cache, g, make_kv, scattered_tables
    K, ref, H = Kernels(verbose=False), ReferenceKernels(compute=torch.float64), 256
    lens = ([1, 450, 1300, 64, 65, 129, 128, 17, 900, 577, 2048])[:rows]
    slots = list(range(rows, 0, -1))
    tables, n_pages, width = scattered_tables(lens, slots, 64, seed=hd)
    cpu, gpu = make_kv(n_pages, nkv, 64, hd, rows + 1, width, 0, 0, torch.bfloat16, tables)
    for i, (slot, n) in enumerate(zip(slots, lens)):
        fill_cache(cpu, gpu, slot, g(n, nkv, hd, dtype=torch.bfloat16, seed=10 + i), g(n, nkv, hd, dtype=torch.bfloat16, seed=40 + i))
        at = cpu.block_table[slot, (n - 1) // 64]
        cpu.storage[at, :, :, (n - 1) % 64] = float("nan")
    a, w, b = g(rows, H, dtype=torch.bfloat16, seed=1), g((nh + 2 * nkv) * hd, H, dtype=torch.bfloat16, seed=2, scale=1.0 / math.sqrt(H)), torch.zeros((nh + 2 * nkv) * hd)
    w[nh * hd:(nh + 1) * hd] = 2.0 * w[:hd]                        # kv head 0's newest key: twice query head 0
    inv = torch.pow(torch.tensor(10000.0, dtype=torch.float64), -2.0 * torch.arange(hd // 2, dtype=torch.float64) / hd).float()
    seqs = [(slot, n - 1, 1) for slot, n in zip(slots, lens)]
    bc, bg = batch_of(seqs, "cpu"), batch_of(seqs, "cuda")
    qkv, kept = (a.double() @ w.double().t()).bfloat16(), cpu.storage.clone()
    q64, want = qkv.double(), torch.empty(rows, nh * hd, dtype=torch.float64)
    ref.rope_append(q64, inv, hd, bc.row_pos, bc.row_seq, bc.seq_slot, bc.seq_len, cpu, nh, nkv, hd)
    ref.attention(q64, cpu, bc, want, nh, nkv, hd, 1.0 / math.sqrt(hd), 0, True)
    for cluster in (1, 2, 4, 8, 16):
        monkeypatch.setattr(Kernels, "_near", lambda *x, c=cluster: c)
        gpu.storage.copy_(kept)
        if rows <= 8:
            row = torch.empty(rows, (nh + 2 * nkv) * hd, dtype=torch.bfloat16, device="cuda")
            args = a.cuda(), w.cuda(), b.cuda(), row, inv.cuda(), bg.row_pos, bg.row_seq, bg.seq_slot, gpu, nh, nkv, hd
        else:
            row = qkv.cuda()
            args = row, inv.cuda(), hd, bg.row_pos, bg.row_seq, bg.seq_slot, bg.seq_len, gpu, nh, nkv, hd
        out = torch.full((rows, nh * hd), 7.0, dtype=torch.bfloat16, device="cuda")
        (K.qkv_rope if rows <= 8 else K.rope_append)(*args)
        K.attention(row, gpu, bg, out, nh, nkv, hd, 1.0 / math.sqrt(hd), 0, True, after_append=True)
        # queries and keys of magnitude 1 to 4 rounded once more than in the statement: scores of magnitude 10 to 4e-2, a weight to 4 %
        got = out.cpu().double()
        assert ((got - want).abs() <= 5e-2 * want.abs().clamp(min=1.0)).all(), (cluster, (got - want).abs().max().item())
