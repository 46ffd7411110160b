"""GPU: the sampler's clusters of CTAs per row, its candidate list and its ordered path, against the oracle's candidate order."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from teenygrad_b200 import ops as o
    return o


def rows_of(kind, rows, cols, g):
    x = torch.randn(rows, cols, generator=g) * 3
    if kind == "ties":         # a handful of values: thousands of ties at every threshold
        x = x.round().clamp(-2, 2)
    elif kind == "masked":     # fewer live entries than top_k, the rest the type's lowest value
        keep = torch.randint(0, cols, (rows, 9), generator=g)
        low = torch.full_like(x, torch.finfo(torch.bfloat16).min)
        x = low.scatter(1, keep, x.gather(1, keep))
    elif kind == "infinite":
        x = x.masked_fill(torch.rand(rows, cols, generator=g) < 0.5, -float("inf"))
    elif kind == "equal":
        x = torch.ones(rows, cols)
    return x.bfloat16()


@pytest.mark.parametrize("kind", ["random", "ties", "masked", "infinite", "equal"])
@pytest.mark.parametrize("rows,cols,top_k", [(1, 151936, 50), (3, 100001, 1024), (37, 33000, 64), (150, 8200, 7), (2, 40, 64), (20, 70000, 1)])
def test_picks_follow_the_definition(ops, kind, rows, cols, top_k):
    from oracle import sampling as osamp
    g = torch.Generator().manual_seed(rows + cols + top_k)
    logits = rows_of(kind, rows, cols, g)
    u = torch.rand(rows, generator=g)
    for pad in (0, 8 - cols % 8, 3):  # contiguous, rows on 16-byte boundaries, rows on none
        buf = torch.full((rows, cols + pad), 100.0, dtype=torch.bfloat16)
        buf[:, :cols] = logits
        got, prob = ops.sample_top_k_top_p(buf.cuda()[:, :cols], 0.8, top_k, 0.9, u.cuda(), want_prob=True)
        got, prob, lf = got.cpu().numpy(), prob.cpu().numpy(), logits.float().numpy()
        for r in list(range(rows))[:8]:
            want, wprob, c, n, cand = osamp.sample_row(lf[r], 0.8, top_k, 0.9, float(u[r]))
            if got[r] == want:
                assert abs(prob[r] - wprob) <= 1e-4 * max(1.0, wprob)
                continue
            # an exponential differs by a few ulps between the GPU and numpy: the neighbour across a boundary of the running sums,
            # or of the nucleus, within 1e-5 of it
            cl = list(cand)
            assert got[r] in cl
            i = cl.index(got[r])
            tol = 1e-5 * c[-1]
            masses = [c[m] for m in range(len(c)) if abs(c[m] - 0.9 * c[-1]) <= tol] + [c[n - 1]]
            assert any((c[i - 1] if i else 0.0) - tol <= float(u[r]) * m <= c[i] + tol for m in masses)
    assert ops.device_error() == 0


def test_candidates_at_the_edges_of_the_bounds(ops):
    """Top-k around what the threads' largest keys bound (a CTA's 1024 threads, one to four CTAs a row), ordered rows, rows whose largest entries share a
    thread, keys far apart, and candidate counts around the two ways of sorting them: the picks of u near 0 and 1 and of the whole nucleus."""
    from oracle import sampling as osamp
    g = torch.Generator().manual_seed(3)
    for rows, cols, top_k in [(3, 33001, 819), (2, 70008, 820), (1, 151936, 1000), (40, 99999, 128), (2, 8200, 129), (2, 1029, 103), (2, 1031, 1024), (80, 16384, 300)]:
        x = torch.randn(rows, cols, generator=g) * 3
        x[0] = x[0].sort().values          # the largest side by side
        x[-1, ::997] *= 2.0 ** 40          # keys far apart
        x = x.bfloat16()
        for u in (0.0, 0.5, 0.999):
            got, prob = ops.sample_top_k_top_p(x.cuda(), 0.9, top_k, 1.0, torch.full((rows,), u).cuda(), want_prob=True)
            for r in {0, rows - 1, rows // 2}:
                want, wprob, c, n, cand = osamp.sample_row(x[r].float().numpy(), 0.9, top_k, 1.0, u)
                if int(got[r]) != want:  # the neighbour across a boundary of the running sums
                    i = list(cand).index(int(got[r]))
                    tol = 1e-5 * c[-1]
                    assert (c[i - 1] if i else 0.0) - tol <= u * c[-1] <= c[i] + tol
                else:
                    assert abs(float(prob[r]) - wprob) <= 1e-4
    assert ops.device_error() == 0
