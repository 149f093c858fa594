"""GPU: attention over cached latent rows in the kernel of latents in blocks of 128 columns (tcgen05), against float64.

Sizes where it can go wrong: one head and a head past each of its widths (16, 32, 64) and past one block of heads; every number of latent blocks;
rotated parts of 16 to 64 columns; a pool row wider than what it holds; more rows than threads of a CTA; a row cut over many CTAs."""
import pytest
import torch

from oracle import berilix_oracle as orc
from tests.test_gpu_hybrid_ops import TOL, close, gen, hops, i32, latent_ref, paged, rnd, status

pytestmark = pytest.mark.gpu
T = torch.bfloat16


def run(H, r, rot, lens, where, seed, extra=0, scale=None):
    """Rows at (sequence, position) `where`; in every row one key outweighs the others for the first head."""
    g = gen(seed)
    total = sum(lens)
    rows = rnd(g, total, r + rot, dtype=T)
    off = [sum(lens[:i]) for i in range(len(lens))]
    n, qo = len(where), 24
    q_abs, q = rnd(g, n, H, r, dtype=T), rnd(g, n, H, qo + rot + 8, dtype=T)
    for t, (s, p) in enumerate(where):
        q_abs[t, 0] = rows[off[s] + [0, p // 2, max(p - 1, 0), p][t % 4], :r] * 3.0
    gate = rnd(g, n, H + 4, dtype=T)
    wide = torch.cat([rows, torch.zeros(total, extra, dtype=T)], 1) if extra else rows
    pool, table = paged(wide, lens, seed)
    pos = torch.tensor([p for _, p in where])
    ang = pos.double()[:, None] * 30.0 ** (-torch.arange(0, rot, 2, dtype=torch.float64) / rot)
    st, scale = status(), scale or 1.5 * (r + rot) ** -0.5
    args = (q_abs.cuda(), q.cuda(), qo, ang.cos().float().cuda(), ang.sin().float().cuda(), pool, table, i32(*[s for s, _ in where]), i32(*pos.tolist()))
    qr = orc.rotate(q.double()[..., qo:qo + rot], pos, 30.0, rot).to(T).double().cuda()
    rows = rows.double().cuda()
    ref = torch.stack([latent_ref(q_abs[t].double().cuda(), qr[t], rows[off[s]:off[s] + p + 1], r, scale) for t, (s, p) in enumerate(where)]).cpu()
    h = hops()
    close(h.latent_attention(*args, gate.cuda()[:, 4:], r, rot, scale, st), ref * orc.sigmoid(gate.double()[:, 4:])[..., None], TOL[T])
    close(h.latent_attention(*args, None, r, rot, scale, st), ref, TOL[T])
    assert int(st) == 0


AROUND = [(0, 0), (1, 14), (2, 15), (3, 16), (4, 62), (4, 63), (5, 64), (6, 129), (6, 100), (6, 2), (7, 699), (7, 400)]
LENS = [1, 15, 16, 17, 64, 65, 130, 700]


@pytest.mark.parametrize("H,r,rot", [(1, 128, 16), (16, 128, 64), (17, 256, 32), (33, 256, 48), (8, 384, 64), (32, 384, 16), (64, 384, 32), (16, 512, 64),
                                     (31, 512, 64), (48, 512, 32), (64, 512, 64), (65, 512, 64), (130, 256, 64)])
def test_tiles_and_heads(H, r, rot):
    run(H, r, rot, LENS, AROUND, H)


@pytest.mark.parametrize("H,r,rot,extra", [(8, 128, 32, 8), (32, 512, 48, 72), (64, 256, 64, 0)])
def test_wider_pool_rows(H, r, rot, extra):
    run(H, r, rot, LENS, AROUND, H + 1, extra=extra)


@pytest.mark.parametrize("H,r", [(16, 256), (32, 512), (33, 512), (64, 256), (65, 512)])
def test_more_rows_than_threads(H, r):
    """Every position of a sequence as a row of its own: 700 rows of 1 to 11 tiles, most of them whole within a CTA.  So many that 33 heads and more come
    in blocks of 64; in the other tests in blocks of 32."""
    run(H, r, 64, [3, 700], [(1, p) for p in range(700)] + [(0, 2)], 5)


@pytest.mark.parametrize("H,r", [(8, 128), (32, 512), (64, 512)])
def test_one_row_over_many_ctas(H, r):
    """Two long rows: every CTA has a piece of a tile or two.  Peaked scores, so that most pieces' weights vanish in the merge."""
    run(H, r, 64, [9000, 4097], [(0, 8999), (1, 4096)], 6)
    run(H, r, 64, [9000, 4097], [(0, 8999), (1, 4096)], 7, scale=0.3)


def test_a_row_without_keys_and_pages_outside_the_pool():
    """A position below zero gives zeros and sets the status, as a page outside the pool does."""
    h, st = hops(), status()
    pool, table = paged(torch.randn(40, 192).to(T), [40], 0)
    z = lambda *s: torch.randn(*s, device="cuda").to(T)
    ones = torch.ones(2, 32, device="cuda")
    out = h.latent_attention(z(2, 4, 128), z(2, 4, 64), 0, ones, ones, pool, table, i32(0, 0), i32(39, -1), None, 128, 64, 1.0, st)
    assert int(st) == 2 and torch.isfinite(out).all() and not out[1].any()
    st.zero_()
    bad = table.clone()
    bad[0, 1] = pool.size(0) + 3
    h.latent_attention(z(1, 4, 128), z(1, 4, 64), 0, ones[:1], ones[:1], pool, bad, i32(0), i32(39), None, 128, 64, 1.0, st)
    assert int(st) == 2


def test_captured():
    """The call in a CUDA graph, replayed on new inputs in the same buffers."""
    g, h, st = gen(1), hops(), status()
    pool, table = paged(rnd(g, 300, 576, dtype=T), [300], 1)
    q_abs, q = rnd(g, 1, 32, 512, dtype=T).cuda(), rnd(g, 1, 32, 64, dtype=T).cuda()
    ones, pos = torch.ones(1, 32, device="cuda"), i32(299)
    call = lambda: h.latent_attention(q_abs, q, 0, ones, ones, pool, table, i0, pos, None, 512, 64, 0.05, st)
    i0 = i32(0)
    call()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = call()
    q_abs.copy_(rnd(g, 1, 32, 512, dtype=T))
    pos.fill_(150)
    graph.replay()
    assert torch.equal(out, call()) and int(st) == 0


SHORT = [1, 63, 64, 200, 256]


@pytest.mark.parametrize("H,r,rot", [(1, 256, 32), (8, 512, 64), (16, 384, 64), (33, 128, 16), (64, 128, 64), (64, 512, 64)])
@pytest.mark.parametrize("lens,rows", [([40, 64, 1, 63], 40), ([40, 64, 1, 63], 166), ([40, 64, 1, 63], 167), (SHORT, 20), (SHORT, 41), (SHORT, 42), ([257, 30], 3)])
def test_short_tables(lens, rows, H, r, rot):
    """Either side of the line up to which the mma.sync kernel has the short contexts (on 148 SMs: 166 tiles of a table of up to 16 blocks)."""
    run(H, r, rot, lens, [(t % len(lens), (7 * t) % lens[t % len(lens)]) for t in range(rows)], rows + H)


@pytest.mark.parametrize("rows,longest", [(19, 8193), (20, 8193), (19, 8192)])
def test_few_rows_behind_a_wide_table(rows, longest):
    """64 heads: fewer than 20 rows behind a table of more than 512 blocks come in blocks of 32 heads."""
    run(64, 512, 64, [longest, 300], [(t % 2, 11 * t) for t in range(rows - 1)] + [(0, longest - 1)], rows)
