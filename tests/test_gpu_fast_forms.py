"""Kernels that have a fast form for aligned or common sizes: the fast form against the general one, or against 64-bit
sums, at the sizes where a tile ends, a remainder begins or the rule changes over."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def K():
    from servelab_b200.ops import kernels
    return kernels


def gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


# ------------------------------------------------- float32 product in 16-byte pieces
@pytest.mark.parametrize("M", [1, 15, 16, 17, 33, 64, 65, 257])
@pytest.mark.parametrize("N,Kd", [(1, 4), (63, 36), (64, 64), (130, 100), (1152, 896), (9728, 32)])
def test_float32_product_is_that_of_the_plain_kernel(M, N, Kd):
    """Rows of a width that is no multiple of 4 go to the plain kernel: the same bits, since both add in k order."""
    g = gen(M * 7 + N)
    a, w = torch.randn(M, Kd + 4, device=DEV, generator=g), torch.randn(N, Kd + 4, device=DEV, generator=g)
    bias = torch.randn(N, device=DEV, generator=g)
    wide_a, wide_w = torch.empty(M, Kd + 5, device=DEV), torch.empty(N, Kd + 5, device=DEV)
    wide_a[:, 1:], wide_w[:, 1:] = a, w
    for b in (None, bias):
        fast, plain = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
        K().gemm_simt(a[:, :Kd], w[:, :Kd], fast, b)
        K().gemm_simt(wide_a[:, 1:Kd + 1], wide_w[:, 1:Kd + 1], plain, b)
        assert torch.equal(fast, plain)
    # three products at once, a row's batches side by side (as the heads of a layer lie)
    heads_a, heads_w = torch.randn(M, 3, Kd, device=DEV, generator=g), torch.randn(3, N, Kd, device=DEV, generator=g)
    out = torch.empty(M, 3, N, device=DEV)
    K().gemm_simt_batched(heads_a, heads_w, out)
    one = torch.empty(M, N, device=DEV)
    for h in range(3):
        K().gemm_simt(heads_a[:, h].contiguous(), heads_w[h], one)
        assert torch.equal(out[:, h], one)


def step(lens, starts=None, page=16, slots=None):
    """A packed step of requests with the given tokens, pages in order."""
    from servelab_b200.engine.batch import BatchEntry, StepContext
    starts = starts or [0] * len(lens)
    entries, at = [], 0
    for i, (n, s) in enumerate(zip(lens, starts)):
        pages = -(-(s + n) // page)
        entries.append(BatchEntry(tokens=[0] * n, start=s, want=(), block_tables=[list(range(at, at + pages))],
                                  state_slot=slots[i] if slots else i))
        at += pages
    return StepContext.pack(entries, 1, DEV), at


def odd_view(t):
    """The same rows at an address and a row stride that 16-byte accesses do not take."""
    wide = torch.zeros(t.shape[0], t.shape[1] + 3, dtype=t.dtype, device=t.device)
    wide[:, 1:1 + t.shape[1]] = t
    return wide[:, 1:1 + t.shape[1]]


# ---------------------------------------- heads' norms, rotation and cache write in pieces
HEADS = {   # q heads, kv heads, key size, value size, rotated, halves, norm, unit norm, row norm, biases, mixed values
    "rotated_halves": (16, 4, 128, 128, 64, True, 0, 0, False, False, None),
    "normed_pairs": (6, 2, 64, 32, 48, False, 64, 0, False, False, "mix"),
    "part_normed_kept": (3, 3, 96, 64, 16, False, 40, 0, False, True, "keep"),
    "unit_after_rotation": (8, 1, 256, 512, 256, True, 0, 256, False, False, None),
    "row_normed_biases": (16, 4, 128, 64, 0, False, 0, 0, True, True, None),
    "row_normed_wide": (40, 8, 96, 64, 0, False, 0, 0, True, True, None),
    "many_heads": (40, 8, 128, 128, 128, True, 128, 0, False, True, None),
}


@pytest.mark.parametrize("name", HEADS)
@pytest.mark.parametrize("lens", [[1], [3, 1, 40], [700], [1100]])
def test_heads_in_pieces_are_those_of_the_general_kernel(name, lens):
    """The general kernel runs on rows at odd addresses; both work in float32 and differ in the order of a head's sum
    of squares: one rounding to bfloat16 (2^-8 of a value) and 2^-16 of the largest where a rotation cancels."""
    H, G, D, Dv, rot, halves, norm, unit, row, biased, mixed = HEADS[name]
    g = gen(len(lens) + H)
    ctx, pages = step(lens, [7 * i for i in range(len(lens))])
    T, width = sum(lens), H * D + G * (D + Dv)
    proj = (torch.randn(T, width, device=DEV, generator=g) * 2).bfloat16()
    nq, nk = (H * D, G * D) if row else (D, D)
    qw, kw = (1 + 0.1 * torch.randn(n, device=DEV, generator=g) for n in (nq, nk))
    bias = [torch.randn(n, device=DEV, generator=g) for n in (H * D, G * D, G * Dv)] if biased else [None] * 3
    freq = 10000.0 ** (-torch.arange(rot // 2, device=DEV) / max(rot // 2, 1)).float()
    first = torch.randn(T, G * Dv, device=DEV, generator=g).bfloat16()
    lam = torch.tensor([0.3], device=DEV)
    got = []
    for p in (proj, odd_view(proj)):
        q = torch.zeros(T, H * D, device=DEV, dtype=torch.bfloat16)
        kc = torch.zeros(pages, G, 16, D, device=DEV, dtype=torch.bfloat16)
        vc = torch.zeros(pages, G, 16, Dv, device=DEV, dtype=torch.bfloat16)
        keep = torch.zeros(T, G * Dv, device=DEV, dtype=torch.bfloat16)
        K().head_prep(p, ctx, ctx.block_tables[0], 16, q_off=0, num_heads=H, q_dim=D, q_norm_w=qw, q_norm_dims=norm,
                      q_rot_off=0, k_off=H * D, num_kv_heads=G, k_dim=D, k_norm_w=kw, k_norm_dims=norm, k_rot_off=0,
                      v_off=H * D + G * D, v_dim=Dv, freq=freq if rot else None, rot_dims=rot, rot_mag=1.1, eps=1e-6,
                      q_out=q, k_cache=kc, v_cache=vc, lam=lam if mixed == "mix" else None,
                      v_first=first if mixed == "mix" else None, v_keep=keep if mixed == "keep" else None,
                      rot_half=halves, q_unit_dims=unit, k_unit_dims=unit, q_bias=bias[0], k_bias=bias[1],
                      v_bias=bias[2], row_norm=row)
        got.append([t.float() for t in (q, kc, vc, keep)])
    assert K().head_prep_status() == 0
    for a, b in zip(*got):
        assert ((a - b).abs() <= b.abs() * 2.0 ** -7 + 2.0 ** -16 * b.abs().max()).all()
    assert got[0][0].abs().max() > 0 and got[0][1].abs().max() > 0 and got[0][2].abs().max() > 0


@pytest.mark.parametrize("biased", [False, True])
@pytest.mark.parametrize("lens", [[2, 30], [600]])
@pytest.mark.parametrize("H,D,rot,R", [(16, 128, 64, 256), (5, 48, 32, 96), (8, 64, 64, 448)])
def test_latent_rows_in_pieces_are_those_of_the_general_kernel(H, D, rot, R, lens, biased):
    """A latent attention's rows: one long key (normed latent, rotated rest), queries whose unrotated part is skipped
    (a bias has that part too)."""
    g = gen(H + len(lens))
    ctx, pages = step(lens)
    T, q_head = sum(lens), D + rot
    proj = torch.randn(T, H * q_head + R + rot, device=DEV, generator=g).bfloat16()
    kw = 1 + 0.1 * torch.randn(R, device=DEV, generator=g)
    freq = 10000.0 ** (-torch.arange(rot // 2, device=DEV) / (rot // 2)).float()
    qb, kb = (torch.randn(n, device=DEV, generator=g) if biased else None for n in (H * q_head, R + rot))
    got = []
    for p in (proj, odd_view(proj)):
        q = torch.zeros(T, H * (R + rot), device=DEV, dtype=torch.bfloat16)
        kc = torch.zeros(pages, 1, 16, R + rot, device=DEV, dtype=torch.bfloat16)
        K().head_prep(p, ctx, ctx.block_tables[0], 16, q_off=0, num_heads=H, q_dim=q_head, q_norm_w=None, q_norm_dims=0,
                      q_rot_off=D, q_out=q[:, R:], q_head_stride=R + rot, q_skip=D, k_off=H * q_head, num_kv_heads=1,
                      k_dim=R + rot, k_norm_w=kw, k_norm_dims=R, k_rot_off=R, v_off=-1, v_dim=0, freq=freq,
                      rot_dims=rot, rot_mag=1.0, eps=1e-6, k_cache=kc, v_cache=None, q_bias=qb, k_bias=kb)
        got.append([q.float(), kc.float()])
    for a, b in zip(*got):
        assert ((a - b).abs() <= b.abs() * 2.0 ** -7 + 2.0 ** -16 * b.abs().max()).all() and a.abs().max() > 0


@pytest.mark.parametrize("T,N,group", [(1, 8, 1), (5, 2048, 1), (300, 1000, 1), (33, 1024, 64)])
def test_sigmoid_gate_in_pieces(T, N, group):
    g = gen(T)
    x, z = (torch.randn(T, n, device=DEV, generator=g).bfloat16() for n in (N, N // group))
    fast, plain = torch.empty_like(x), torch.empty_like(x)
    K().sigmoid_gate(x, z, fast, group)
    K().sigmoid_gate(odd_view(x), odd_view(z), plain, group)
    assert torch.equal(fast, plain)


# ------------------------------------------------------------ convolution, norms with a gate
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("C,lens", [(264, [256]), (264, [1, 2, 300, 7]), (264, [129, 128, 5]), (1032, [3053]),
                                    (1032, [1, 2, 3100, 7]), (520, [6100, 9, 130, 5]), (1032, [129] * 24)])
def test_convolution_of_runs_is_that_of_single_tokens(dtype, taps, C, lens):
    """Long portions of large steps (3 Mi elements, 128 tokens a request) take runs of tokens a thread; other steps, and
    rows at an odd address, the kernel that takes them one by one.  The same products in the same
    order: the same bits, in the rows and in the records."""
    g = gen(taps + len(lens))
    ctx, _ = step(lens)
    T = sum(lens)
    proj = torch.randn(T, C + 8, device=DEV, generator=g).to(dtype)
    w, b_in, b_out = (torch.randn(*s, device=DEV, generator=g) for s in ((taps, C), (C,), (C,)))
    record = torch.randn(len(lens), (taps - 1) * C + 4, device=DEV, generator=g)
    got = []
    for p in (proj, odd_view(proj)):
        out, state = torch.zeros(T, C, device=DEV, dtype=dtype), record.clone()
        K().short_conv(p, w, state, ctx, out, b_in, b_out, activation="silu")
        got.append((out, state))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,groups,size", [(1, 1, 4), (7, 3, 100), (33, 8, 256), (5, 4, 512), (9, 2, 1024), (3, 2, 1028)])
def test_gated_norms_against_64_bits(dtype, T, groups, size):
    """Sums of up to 1,028 squares in float32: 1e-6 of a value, and the result's rounding."""
    g, n = gen(T + size), groups * size
    x, lam, w = (torch.randn(*s, device=DEV, generator=g) for s in ((T, 2 * n), (1,), (n,)))
    gate = torch.randn(T, n, device=DEV, generator=g).to(dtype)
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 4e-6

    def rms(v):
        v = v.reshape(T, groups, size)
        return (v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-6)).reshape(T, n)
    d, z = x.double(), gate.double()
    pairs = d.view(T, groups, 2, size)
    for maps, rows in ((1, d[:, :n]), (2, pairs[:, :, 0] - lam.double() * pairs[:, :, 1])):
        out = torch.empty(T, n, device=DEV, dtype=dtype)
        K().group_norm_gate(x[:, :n] if maps == 1 else x, groups, size, out, eps=1e-6, weight=w, factor=0.7, gate=gate,
                            gate_activation="silu", maps=maps, lam=lam)
        want = 0.7 * rms(rows) * w.double() * z * torch.sigmoid(z)
        assert ((out.double() - want).abs() <= tol * want.abs() + 1e-6).all()
    out = torch.empty(T, n, device=DEV, dtype=dtype)
    K().gate_group_norm(x[:, :n], gate, groups, out, eps=1e-6, weight=w, factor=1.5)
    want = 1.5 * rms(d[:, :n] * z * torch.sigmoid(z)) * w.double()
    assert ((out.double() - want).abs() <= tol * want.abs() + 1e-6).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("size", [4, 100, 256, 512, 1024])
@pytest.mark.parametrize("T", [255, 256, 257])
def test_gate_before_norm_of_many_parts(dtype, size, T):
    """Bfloat16 calls of 2,048 parts and more have a kernel of their own: 64-bit sums (1e-6 of a value and its
    rounding), and the general form on rows at odd addresses (a rounding to bfloat16 apart).  A float32 row is the
    same bits in a call of a few rows."""
    groups, g = 8, gen(T + size)
    n = groups * size
    x, w = torch.randn(T, n, device=DEV, generator=g), torch.randn(n, device=DEV, generator=g)
    gate = torch.randn(T, n, device=DEV, generator=g).to(dtype)

    def run(x, gate):
        out = torch.empty(x.shape[0], n, device=DEV, dtype=dtype)
        K().gate_group_norm(x, gate, groups, out, eps=1e-6, weight=w, factor=1.5)
        return out
    out, z = run(x, gate), gate.double()
    v = (x.double() * z * torch.sigmoid(z)).view(T, groups, size)
    want = 1.5 * (v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-6)).view(T, n) * w.double()
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 4e-6
    assert ((out.double() - want).abs() <= tol * want.abs() + 1e-6).all()
    odd = run(odd_view(x), odd_view(gate)).double()
    assert ((out.double() - odd).abs() <= 2 * tol * want.abs() + 2e-6).all()
    if dtype == torch.float32:
        assert torch.equal(out[-7:], run(x[-7:], gate[-7:]))


@pytest.mark.parametrize("T,groups,size", [(257, 8, 64), (257, 8, 100), (3, 4, 512), (2, 1, 2048), (2, 3, 4500)])
@pytest.mark.parametrize("act", ["silu", "sigmoid"])
def test_gate_before_norm_is_float32_whatever_the_result(T, groups, size, act):
    """The gated value enters a float32 sum of squares: bfloat16 results are the float32 results rounded, bit for bit (the
    same kernel, the same order of the sums)."""
    g = gen(size)
    n = groups * size
    x, w = torch.randn(T, n, device=DEV, generator=g), torch.randn(n, device=DEV, generator=g)
    gate = (torch.randn(T, n, device=DEV, generator=g) * 6).bfloat16()
    outs = []
    for dtype in (torch.float32, torch.bfloat16):
        out = torch.empty(T, n, device=DEV, dtype=dtype)
        K().gate_group_norm(x, gate.to(dtype), groups, out, eps=1e-6, weight=w, factor=1.5, gate_activation=act)
        outs.append(out.bfloat16())
    assert torch.equal(*outs)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n", [4, 1024, 1028, 2048, 3584, 4100])
def test_sum_of_two_norms_against_64_bits(dtype, n):
    g = gen(n)
    a, b = (torch.randn(5, n, device=DEV, generator=g) * 3 for _ in range(2))
    wa, wb = (torch.randn(n, device=DEV, generator=g) for _ in range(2))
    out = torch.empty(5, n, device=DEV, dtype=dtype)
    K().norm_sum2(a, b, wa, wb, 1e-6, 0.5, out)
    u, v = ((t.double() / torch.sqrt((t.double() ** 2).mean(-1, keepdim=True) + 1e-6)) * w.double()
            for t, w in ((a, wa), (b, wb)))
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 0.0
    assert ((out.double() - 0.5 * (u + v)).abs() <= tol * (u + v).abs() + 2e-6 * (u.abs() + v.abs()) + 1e-7).all()


# ------------------------------------------------------------------------- routed experts
@pytest.mark.parametrize("M,E,Kd", [(512, 32, 2048), (513, 5, 32), (700, 33, 1056), (640, 64, 96)])
def test_router_logits_of_many_tokens(M, E, Kd):
    """Float32 sums of up to 2,048 products, an eighth of them at a time: 3e-7 of the result's norm."""
    g = gen(M + E)
    x, w = torch.randn(M, Kd + 8, device=DEV, generator=g).bfloat16()[:, :Kd], torch.randn(E, Kd, device=DEV, generator=g)
    want = x.double() @ w.double().T
    assert (K().router_logits(x, w).double() - want).norm() <= 1e-6 * want.norm()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,h,I", [(3, 64, 40), (70, 200, 64), (5, 1024, 512)])
def test_small_steps_of_the_experts_take_rows_of_any_stride(T, h, I, dtype):
    """Every second column, and a transposed matrix: the same bits as their copies, in each form of the products."""
    g, E, top = gen(T), 4, 2
    x = torch.randn(T, 2 * h, device=DEV, generator=g).to(dtype)
    wg, wd = ((torch.randn(*s, device=DEV, generator=g) * s[-1] ** -0.5).to(dtype) for s in ((E, 2 * I, h), (E, h, I)))
    ids = torch.stack([torch.randperm(E, device=DEV, generator=g)[:top] for _ in range(T)]).int().contiguous()
    w = torch.rand(T, top, device=DEV, generator=g)
    for view in (x[:, ::2], x[:, :h].T.contiguous().T):
        assert view.stride(1) != 1
        assert torch.equal(K().moe_experts(view, ids, w, wg, wd, None), K().moe_experts(view.contiguous(), ids, w, wg, wd, None))


EXPERTS_FORMS = {"tcgen05": "slb_gemm_rows_experts_bf16", "library": "_grouped_mm", "mma": "slb_moe_gate_up_mma_bf16"}


def experts_form(monkeypatch, form):
    """Leaves routed experts one form of their products; the list it returns names the products that ran."""
    from servelab_b200.ops import library as L
    monkeypatch.setattr(K(), "moe_tcgen05", form == "tcgen05")
    monkeypatch.setattr(K(), "moe_vendor_grouped", form == "library")
    ran = []
    for owner, name in ((L.core(), EXPERTS_FORMS["tcgen05"]), (torch, EXPERTS_FORMS["library"]), (L.core(), EXPERTS_FORMS["mma"])):
        real = getattr(owner, name)
        monkeypatch.setattr(owner, name, lambda *a, real=real, name=name, **kw: ran.append(name) or real(*a, **kw))
    return ran


@pytest.mark.parametrize("form", EXPERTS_FORMS)
def test_large_steps_of_the_experts_take_rows_of_any_stride(monkeypatch, form):
    """Every second column of a wider matrix: the library's products took such rows, and so must the steps that read
    them themselves."""
    g = gen(3)
    x, w = torch.randn(600, 512, device=DEV, generator=g).bfloat16(), torch.randn(16, 512, device=DEV, generator=g)
    want = x[:, ::2].double() @ w[:, ::2].double().T
    for a, b in ((x[:, ::2], w[:, ::2].contiguous()), (x[:, ::2].contiguous(), w[:, ::2])):
        assert (K().router_logits(a, b).double() - want).norm() <= 1e-6 * want.norm()
    T, E, top, h, I = 300, 8, 4, 1024, 2048
    x = torch.randn(T, 2 * h, device=DEV, generator=g).bfloat16()
    wg, wd = ((torch.randn(*s, device=DEV, generator=g) * s[-1] ** -0.5).bfloat16() for s in ((E, 2 * I, h), (E, h, I)))
    ids = torch.stack([torch.randperm(E, device=DEV, generator=g)[:top] for _ in range(T)]).int().contiguous()
    p = torch.rand(T, top, device=DEV, generator=g)
    ran = experts_form(monkeypatch, form)
    packed = K().moe_experts(x[:, ::2].contiguous(), ids, p, wg, wd, None)
    assert set(ran) == {EXPERTS_FORMS[form]}
    wide = K().moe_experts(x[:, ::2], ids, p, wg, wd, None)
    assert torch.equal(wide, packed)


@pytest.mark.parametrize("P,E", [(1, 1), (3, 7), (256, 32), (8191, 32), (64, 1024), (20001, 60)])
def test_plan_of_the_experts_rows(P, E):
    from servelab_b200.ops import library as L
    ids = torch.randint(0, E, (P,), device=DEV, dtype=torch.int32, generator=gen(P))
    lib = L.core()
    plan = torch.full((lib.slb_moe_plan_ints(P, E),), -7, dtype=torch.int32, device=DEV)
    L.check(lib.slb_moe_plan(ids.data_ptr(), P, E, plan.data_ptr(), K()._stream()), "moe_plan")
    rows = lib.slb_moe_tile_rows(P, E)
    tiles = -(-P // rows) + E
    p, counts = plan.cpu().long(), torch.bincount(ids.cpu().long(), minlength=E)
    assert torch.equal(p[:E], counts) and torch.equal(p[E:2 * E + 1], torch.cat([torch.zeros(1, dtype=torch.long), counts.cumsum(0)]))
    at = 3 * E + 1
    want = [(e, r) for e in range(E) for r in range(0, int(counts[e]), rows)]
    got = list(zip(p[at:at + tiles].tolist(), p[at + tiles:at + 2 * tiles].tolist()))
    assert got[:len(want)] == want and all(e == -1 for e, _ in got[len(want):])
    order, where = p[at + 2 * tiles:at + 2 * tiles + P], p[at + 2 * tiles + P:]
    assert len(where) == P and torch.equal(order.sort().values, torch.arange(P)) and torch.equal(where[order], torch.arange(P))
    assert (ids.cpu().long()[order].diff() >= 0).all()


@pytest.mark.parametrize("P,E", [(1, 1), (256, 32), (1000, 32), (1280, 32), (5000, 32)])
def test_plan_of_the_products_on_cuda_cores_has_full_tiles(P, E):
    """One tile an expert up to 64 rows, however few rows the experts get: a smaller tile would cost them as much."""
    from servelab_b200.ops import library as L
    ids = torch.randint(0, E, (P,), device=DEV, dtype=torch.int32, generator=gen(P))
    ids[:P // 3] = 0                                      # a crowded expert
    lib = L.core()
    plan = torch.full((lib.slb_moe_plan_simt_ints(P, E),), -7, dtype=torch.int32, device=DEV)
    L.check(lib.slb_moe_plan_simt(ids.data_ptr(), P, E, plan.data_ptr(), K()._stream()), "moe_plan")
    p, tiles, at = plan.cpu().tolist(), -(-P // 64) + E, 3 * E + 1
    counts = torch.bincount(ids.cpu().long(), minlength=E).tolist()
    want = [(e, r) for e in range(E) for r in range(0, counts[e], 64)]
    got = list(zip(p[at:at + tiles], p[at + tiles:at + 2 * tiles]))
    assert len(p) == at + 2 * tiles + 2 * P
    assert got[:len(want)] == want and all(e == -1 for e, _ in got[len(want):])


@pytest.mark.parametrize("T,E,top,h,I", [(9, 8, 2, 36, 20), (100, 8, 3, 60, 28), (300, 5, 2, 44, 36)])
def test_experts_products_on_cuda_cores(T, E, top, h, I):
    """Float32, few and many rows an expert, one expert with more rows than a tile: sums of at most 60 products in
    order against 64 bits, 2e-6 of the norm."""
    g = gen(T + E)
    x = torch.randn(T, h, device=DEV, generator=g)
    wg, wd = (torch.randn(*s, device=DEV, generator=g) * s[-1] ** -0.5 for s in ((E, 2 * I, h), (E, h, I)))
    ids = torch.stack([torch.randperm(E, device=DEV, generator=g)[:top] for _ in range(T)]).int().contiguous()
    ids[:, 0] = 1
    ids[:, 1:] = torch.where(ids[:, 1:] == 1, 0, ids[:, 1:])
    w = torch.rand(T, top, device=DEV, generator=g)
    gu = torch.einsum("tkih,th->tki", wg.double()[ids.long()], x.double())
    act = gu[..., :I] * torch.sigmoid(gu[..., :I]) * gu[..., I:]
    want = torch.einsum("tk,tkhi,tki->th", w.double(), wd.double()[ids.long()], act)
    assert (K().moe_experts(x, ids, w, wg, wd, None).double() - want).norm() <= 2e-6 * want.norm()


def test_rows_of_a_tile_follow_the_rows_an_expert_gets():
    from servelab_b200.ops import library as L
    rows = L.core().slb_moe_tile_rows
    assert [rows(32 * n, 32) for n in (1, 8, 9, 32, 33, 200)] == [16, 16, 32, 32, 64, 64]
    assert [rows(16 * n, 16) for n in (8, 9, 64, 65)] == [16, 32, 32, 64]


@pytest.mark.parametrize("form", ["tcgen05", "library"])
def test_pairs_without_an_expert_add_nothing_in_large_steps(monkeypatch, form):
    """The list of a plan has an entry for every pair, also where ids are no expert's: in range, and the step's sum is
    that of the other pairs (the zero weights beside valid ids: the same products, the same bits)."""
    from servelab_b200.ops import library as L
    T, E, top, h, I, g = 300, 8, 4, 1024, 2048, gen(5)
    x = torch.randn(T, h, device=DEV, generator=g).bfloat16()
    wg, wd = ((torch.randn(*s, device=DEV, generator=g) * s[-1] ** -0.5).bfloat16() for s in ((E, 2 * I, h), (E, h, I)))
    ids = torch.stack([torch.randperm(E, device=DEV, generator=g)[:top] for _ in range(T)]).int().contiguous()
    w = torch.rand(T, top, device=DEV, generator=g)
    bad = torch.rand(T, top, device=DEV, generator=g) < 0.2
    lib, P = L.core(), T * top
    plan = torch.full((lib.slb_moe_plan_ints(P, E),), -7, dtype=torch.int32, device=DEV)
    holes = torch.where(bad, -1, ids)
    L.check(lib.slb_moe_plan(holes.data_ptr(), P, E, plan.data_ptr(), K()._stream()), "moe_plan")
    order, rows = plan[-2 * P:-P].cpu(), int(plan[2 * E])
    assert rows == P - int(bad.sum()) and (order[rows:] == 0).all()
    assert torch.equal(order[:rows].sort().values, (~bad).view(-1).nonzero().view(-1).int().cpu())
    ran = experts_form(monkeypatch, form)
    for weighted in (False, True):
        got = K().moe_experts(x, holes, w, wg, wd, None, weight_inputs=weighted)
        want = K().moe_experts(x, ids, torch.where(bad, 0.0, w), wg, wd, None, weight_inputs=weighted)
        assert torch.equal(got, want)
    assert set(ran) == {EXPERTS_FORMS[form]}


@pytest.mark.parametrize("T,E,top,h,I", [(1, 8, 2, 64, 40), (3, 4, 4, 128, 72), (33, 8, 2, 200, 64), (64, 8, 2, 64, 136),
                                         (100, 5, 3, 72, 64), (300, 4, 2, 128, 64)])
def test_experts_products_at_few_and_many_rows(T, E, top, h, I):
    """Tiles of 16, 32 and 64 rows (up to 8, 64 and more rows of a few experts) against 64 bits: two roundings to bfloat16 of
    the first product, one of the activation, one of the result."""
    g = gen(T)
    x = torch.randn(T, h, device=DEV, generator=g).bfloat16()
    wg, wd = ((torch.randn(*s, device=DEV, generator=g) * s[-1] ** -0.5).bfloat16() for s in ((E, 2 * I, h), (E, h, I)))
    ids = torch.stack([torch.randperm(E, device=DEV, generator=g)[:top] for _ in range(T)]).int().contiguous()
    if T > 50:
        ids[:, 0] = 1                                     # one expert with more rows than a tile
        ids[:, 1:] = torch.where(ids[:, 1:] == 1, 0, ids[:, 1:])
    w = torch.rand(T, top, device=DEV, generator=g)
    got = K().moe_experts(x, ids, w, wg, wd, None).double()
    want = torch.zeros_like(got)
    for t in range(T):
        for k in range(top):
            e = int(ids[t, k])
            gu = wg[e].double() @ x[t].double()
            act = gu[:I] * torch.sigmoid(gu[:I]) * gu[I:]
            want[t] += w[t, k].double() * (wd[e].double() @ act)
    assert (got - want).norm() <= 2.0 ** -7 * want.norm()


# ------------------------------------------------------- state space in chunks
@pytest.mark.parametrize("lens", [[17], [63, 64], [65, 16, 200], [130, 1, 700]])
@pytest.mark.parametrize("H,P,N,G", [(4, 64, 128, 2), (2, 72, 64, 1), (3, 8, 64, 3), (2, 136, 128, 1)])
def test_chunks_in_pieces_are_those_of_the_general_kernels(H, P, N, G, lens):
    """Rows at an odd address go to the general kernels, whose weighted x is rounded in another order before its split
    (2^-17 of every term)."""
    _chunks_in_pieces(H, P, N, G, lens)


@pytest.mark.parametrize("lens", [[700, 65, 1300], [2000], [64] * 40 + [1]])
@pytest.mark.parametrize("H,P,N,G", [(48, 64, 128, 2), (20, 136, 64, 1), (33, 64, 64, 1), (128, 8, 128, 1)])
def test_blocks_of_several_heads_are_those_of_the_general_kernels(H, P, N, G, lens):
    """Sizes whose blocks take two heads and more, a remainder of heads at the end of a group, heads of several blocks of
    columns."""
    _chunks_in_pieces(H, P, N, G, lens)


@pytest.mark.parametrize("H,N,odd,lens,launches", [(32, 64, False, [64] * 20, 2), (32, 128, False, [100], 2), (4, 64, False, [2000], 3),
                                                   (4, 64, True, [64] * 20, 3), (4, 96, False, [100], 3)])
def test_launches_of_the_chunks_are_counted(H, N, odd, lens, launches):
    """Walk and outputs; sums, scan and outputs; the general form on rows at an odd address and for other state sizes."""
    from torch.profiler import ProfilerActivity, profile
    P, T, g = 64, sum(lens), gen(N)
    ctx, _ = step(lens)
    u = torch.randn(T, H * P + 2 * N, device=DEV, generator=g).bfloat16()
    u = odd_view(u) if odd else u
    dt, state, out = torch.zeros(T, H, device=DEV), torch.zeros(len(lens), H * N * P, device=DEV), torch.zeros(T, H * P, device=DEV)
    one = torch.ones(H, device=DEV)

    def run():
        K().state_space(ctx, u, dt, state, out, num_heads=H, value_dim=P, state_dim=N, groups=1, dt_bias=one, rate=one, skip=one)
    run()
    before = K().launch_count
    with profile(activities=[ProfilerActivity.CUDA]) as seen:
        run()
        torch.cuda.synchronize()
    kernels = sum(e.count for e in seen.key_averages() if "state_chunk" in e.key)
    assert K().launch_count - before == launches == kernels


def _chunks_in_pieces(H, P, N, G, lens):
    g, T = gen(H + len(lens)), sum(lens)
    ctx, _ = step(lens)
    rows = torch.randn(T, H * P + 2 * G * N, device=DEV, generator=g).bfloat16()
    dt, bias = torch.randn(T, H, device=DEV, generator=g) - 2, torch.randn(H, device=DEV, generator=g)
    rate, skip = torch.rand(H, device=DEV, generator=g) * 4 + 0.1, torch.randn(H, device=DEV, generator=g)
    record = torch.randn(len(lens), H * N * P + 4, device=DEV, generator=g)
    got = []
    for u in (rows, odd_view(rows)):
        state, out = record.clone(), torch.zeros(T, H * P, device=DEV)
        K().state_space(ctx, u, dt, state, out, num_heads=H, value_dim=P, state_dim=N, groups=G, dt_bias=bias, rate=rate,
                        skip=skip)
        got.append((out, state))
    for a, b in zip(*got):
        assert (a - b).norm() <= 2.0 ** -17 * b.norm() and b.norm() > 0


# ------------------------------------------------ activation in the cluster product's epilogue
@pytest.mark.parametrize("M", [1, 2, 16, 17, 40, 64])
@pytest.mark.parametrize("inter,Kd,splits", [(64, 512, 2), (192, 1024, 8), (128, 520, 3)])
def test_cluster_product_with_activation_is_product_then_activation(M, inter, Kd, splits):
    g = gen(M + inter)
    x, w = torch.randn(M, Kd, device=DEV, generator=g).bfloat16(), (torch.randn(2 * inter, Kd, device=DEV, generator=g) * 0.05).bfloat16()
    fused = K().gemm_tc_cluster(x, w, splits=splits, swiglu=True)
    gu, act = K().gemm_tc_cluster(x, w, splits=splits), torch.empty(M, inter, device=DEV, dtype=torch.bfloat16)
    K().swiglu(gu, act, K().SWIGLU_BLOCK)
    assert torch.equal(fused, act) and act.float().abs().max() > 0
    assert K().gemm_tc_status() == 0


@pytest.mark.parametrize("D", [60, 64, 68, 128])
@pytest.mark.parametrize("Hh,Dv", [(1, 8), (2, 20), (6, 200)])
def test_walk_over_the_chunks_against_the_recurrence(D, Hh, Dv):
    """Both widths of a slice of value columns (few and many slices in the launch), the key sizes with loops of
    fixed length and their neighbours.  float32 sums of at most 70 x D products against 64 bits: 3e-5 of the
    largest value, the bound the other sizes are held to."""
    import test_gpu_sumolorn as case
    from servelab_b200.ops import kernels
    lens = [31, 32, 70]
    proj, z, bias = case._gated_case(5, Hh, D, Dv, sum(lens), torch.bfloat16, z_shift=1.0)
    want = case._gated_want(proj, z, bias, Hh, D, Dv, lens, 4.0, D ** -0.5)
    state = torch.zeros(3, Hh * D * Dv, device="cuda")
    out = case._run_gated_chunked(kernels, proj.cuda(), z.cuda(), bias.cuda(), state, Hh, D, Dv,
                                  [[(0, 0, 31), (1, 31, 32), (2, 63, 70)]], 4.0, D ** -0.5)
    assert (out.double().cpu() - want).abs().max() < 3e-5 * max(1.0, float(want.abs().max()))


@pytest.mark.parametrize("D,Dv", [(60, 200), (64, 64), (128, 20), (132, 72), (256, 8)])
@pytest.mark.parametrize("lens", [[31, 32, 70], [600]])
def test_chunks_side_by_side_against_the_recurrence(monkeypatch, D, Dv, lens):
    """The form without a walk over the chunks (up to 128 and more state rows a block, slices of values that end
    anywhere, more chunks than the scan loads at once), to the bound that the walk is held to; the records it leaves
    are the walk's bits, whose sums have the same order."""
    import test_gpu_sumolorn as case
    from servelab_b200.ops import kernels
    H, T = 2, sum(lens)
    proj, z, bias = case._gated_case(5, H, D, Dv, T, torch.bfloat16, z_shift=1.0)
    want = case._gated_want(proj, z, bias, H, D, Dv, lens, 4.0, D ** -0.5)
    at, parts = 0, []
    for i, n in enumerate(lens):
        parts.append((i, at, n))
        at += n
    states = []
    for form in (True, False):
        monkeypatch.setattr(kernels, "force_side_by_side", form)
        states.append(torch.zeros(len(lens), H * D * Dv, device="cuda"))
        out = case._run_gated_chunked(kernels, proj.cuda(), z.cuda(), bias.cuda(), states[-1], H, D, Dv, [parts], 4.0,
                                      D ** -0.5)
        assert (out.double().cpu() - want).abs().max() < 3e-5 * max(1.0, float(want.abs().max()))
    assert torch.equal(*states)


def test_long_requests_of_few_values_have_their_chunks_side_by_side():
    """The points at which both forms were measured, chunks of 32 tokens."""
    from servelab_b200.ops import library as L
    rule = L.core().slb_decay_gated_chunk_side_by_side
    assert all(rule(*p) for p in ((64, 1, 4, 64, 128), (32, 1, 2, 64, 64), (32, 1, 1, 128, 128), (256, 1, 8, 64, 64),
                                  (64, 2, 1, 128, 128)))
    assert not any(rule(*p) for p in ((16, 1, 4, 64, 128), (16, 1, 1, 128, 128), (64, 1, 8, 128, 256), (64, 1, 16, 128, 128),
                                      (256, 1, 8, 128, 256), (127, 64, 4, 64, 128), (64, 64, 1, 64, 64), (512, 64, 8, 64, 64)))


@pytest.mark.parametrize("D,Dv", [(64, 64), (128, 40), (192, 64)])
def test_scans_over_chunks_report_waits_that_gave_up(D, Dv):
    """Two and one record a block (key sizes up to 128 and above), requests of one and of several chunks: no wait
    gives up, every row is written."""
    lens, H, g = [32, 70, 129], 2, gen(D)
    ctx, _ = step(lens)
    T = sum(lens)
    proj = torch.randn(T, H * (3 * D + 2 * Dv), device=DEV, generator=g).bfloat16()
    z, bias, norm = (torch.randn(*s, device=DEV, generator=g) for s in ((T, H * D), (H * D,), (H * Dv,)))
    out = torch.full((T, H * Dv), float("nan"), device=DEV, dtype=torch.bfloat16)
    K().delta_rule(ctx, proj, torch.zeros(3, H * D * Dv, device=DEV), out, r_off=0, k_off=H * D, v_off=2 * H * D,
                   a_off=H * (2 * D + Dv), g_off=H * (3 * D + Dv), num_heads=H, head_dim=D, value_dim=Dv, a_bias=bias,
                   gate_z=z, decay_coef=0.6, unit_eps=1e-6, norm_w=norm, norm_eps=1e-5)
    rows = torch.full((T, H * Dv), float("nan"), device=DEV)
    K().decay_attention(proj, ctx, torch.zeros(3, H * D * Dv, device=DEV), None, rows, q_off=0, k_off=H * D, v_off=2 * H * D,
                        num_heads=H, head_dim=D, value_dim=Dv, gate_z=z, gate_tau=4.0)
    assert out.isfinite().all() and rows.isfinite().all()
    assert K().delta_chunk_status() == 0 and K().decay_gated_chunk_status() == 0


# ----------------------------------------------------- more splits in decode steps, and their error
@pytest.mark.parametrize("N,Kd", [(896, 896), (640, 1152), (896, 4864)])
def test_finer_k_splits_are_no_less_exact(N, Kd):
    """Ten inputs, the chosen splits against one: float32 sums in another order under the same rounding to bfloat16,
    which makes nearly all of the error."""
    assert K().tc_cluster_splits(N, Kd) > 5
    total = {0: 0.0, 1: 0.0}
    for seed in range(10):
        g = gen(seed)
        x, w = torch.randn(3, Kd, device=DEV, generator=g).bfloat16(), (torch.randn(N, Kd, device=DEV, generator=g) * 0.05).bfloat16()
        want = x.double() @ w.double().T
        for splits in total:
            total[splits] += float((K().gemm_tc_cluster(x, w, splits=splits).double() - want).norm() / want.norm())
    assert total[0] <= 1.005 * total[1] and total[1] < 10 * 2.0 ** -8


@pytest.mark.parametrize("H,G,D", [(14, 2, 64), (28, 4, 128)])
def test_split_requests_of_five_tiles_are_no_less_exact(monkeypatch, H, G, D):
    """Ten inputs, 8 requests of 270 to 384 keys, the chosen splits against none: the same keys with the largest score
    of a split in place of the request's; the probabilities' and the result's rounding make the error."""
    lens = [270, 300, 319, 320, 321, 350, 383, 384]
    ctx, pages = step([1] * 8, [n - 1 for n in lens])
    assert K().decode_ws_unsplit(8, G, H // G, D) < 5
    total = {0: 0.0, 1: 0.0}
    for seed in range(10):
        g = gen(seed)
        q, kc, vc = (torch.randn(*s, device=DEV, generator=g).bfloat16() for s in ((8, H * D), (pages, G, 16, D), (pages, G, 16, D)))
        want, at = [], 0
        for i, n in enumerate(lens):
            used = -(-n // 16)
            k, v = (c[at:at + used].transpose(0, 1).reshape(G, used * 16, D)[:, :n].double() for c in (kc, vc))
            p = torch.softmax(q[i].double().view(G, H // G, D) @ k.transpose(1, 2) * D ** -0.5, -1)
            want.append((p @ v).reshape(-1))
            at += used
        want = torch.stack(want)
        for splits in total:
            monkeypatch.setattr(K(), "decode_ws_force_splits", splits)
            out = torch.empty(8, H * D, device=DEV, dtype=torch.bfloat16)
            K().decode_attention(ctx, q, kc, vc, out, ctx.block_tables[0], H, G, D, 16, D ** -0.5, 0)
            total[splits] += float((out.double() - want).norm() / want.norm())
    assert total[0] <= 1.03 * total[1] and total[1] < 10 * 2.0 ** -7
    assert K().decode_attention_status(D) == 0


# ------------------------------------------------------------- products of a feed-forward over many tokens
def _act64(g, u, act):
    if act == "gelu_tanh":
        return torch.nn.functional.gelu(g, approximate="tanh") * u
    if act == "swish_clamped":
        g, u = g.clamp(max=1.3), u.clamp(-1.3, 1.3) + 1
        return g * torch.sigmoid(1.7 * g) * u
    return g * torch.sigmoid(g) * u


@pytest.mark.parametrize("act", ["silu", "gelu_tanh", "swish_clamped"])
@pytest.mark.parametrize("T,I,Kd,block,nt", [(1, 64, 8, 64, 0), (33, 64, 64, 64, 32), (257, 192, 200, 64, 96), (300, 112, 72, 0, 256),
                                             (700, 16, 128, 0, 160), (2048, 4864, 896, 64, 0), (480, 1408, 2048, 0, 0)])
def test_gated_product_of_many_tokens(T, I, Kd, block, nt, act):
    """Against 64 bits, in tiles that do not divide tokens, features or K: the result is rounded once (2^-9 relative), and
    float32 sums of K products and a hardware exponential and reciprocal before it change it by less than a quarter of
    that: 2.5e-3 of the norm."""
    g = gen(T + I)
    x = torch.randn(T, Kd, device=DEV, generator=g).bfloat16()
    w = (torch.randn(2 * I, Kd, device=DEV, generator=g) * Kd ** -0.5).bfloat16()
    assert K().gemm_rows_gated_takes(x, w, block)
    got = K().gemm_rows_gated(x, w, block, act, 1.3, 1.7, tile_tokens=nt).double()
    y = x.double() @ w.double().T
    gu = y.view(T, I // 64, 2, 64).transpose(1, 2).reshape(T, 2, I) if block else y.view(T, 2, I)
    want = _act64(gu[:, 0], gu[:, 1], act)
    assert (got - want).norm() <= 2.5e-3 * want.norm() and K().gemm_rows_status() == 0


@pytest.mark.parametrize("T", [129, 300])
@pytest.mark.parametrize("block", [0, 64])
def test_gated_linear_takes_rows_that_overlap(T, block):
    """A broadcast row and rows 8 elements apart: what their copies give, to the rounding of a second kernel (gate and up
    rounded to bfloat16 first, 2^-8 of the norm)."""
    from servelab_b200.ops import linear
    g = gen(T)
    buf, w = torch.randn(8 * T + 512, device=DEV, generator=g).bfloat16(), (torch.randn(2048, 512, device=DEV, generator=g) * 0.04).bfloat16()
    assert K().gemm_rows_gated_pays(T, 1024, 512)
    for x in (buf[:512].expand(T, 512), buf.as_strided((T, 512), (8, 1))):
        got, want = linear.gated_linear(x, w, block), linear.gated_linear(x.contiguous(), w, block)
        assert (got.double() - want.double()).norm() <= 2.0 ** -8 * want.double().norm()


@pytest.mark.parametrize("counts", [[0, 1, 300, 33], [256, 257, 0, 17, 513, 1, 2, 31], [700, 2400, 5], [0, 0, 1]])
@pytest.mark.parametrize("weighted", [False, True])
def test_experts_products_over_sorted_rows(counts, weighted):
    """Experts without rows, with one, with whole tiles and one more; both results of the second product; rows of no
    expert stay as they are.  Bound as above (float32 rows: 2^-20 for sums of 112 products)."""
    from servelab_b200.ops import library as L
    g, E, h, I = gen(sum(counts)), len(counts), 72, 112
    P = sum(counts) + 5
    offs = torch.tensor([0] + counts, device=DEV).cumsum(0).int()
    x = torch.randn(P, h, device=DEV, generator=g).bfloat16()
    wg, wd = ((torch.randn(*s, device=DEV, generator=g) * s[-1] ** -0.5).bfloat16() for s in ((E, 2 * I, h), (E, h, I)))
    order, rw = torch.randperm(P, device=DEV, generator=g).int(), torch.rand(P, device=DEV, generator=g)
    act = torch.full((P, I), float("nan"), device=DEV, dtype=torch.bfloat16)
    lib, st = L.core(), K()._stream()
    L.check(lib.slb_gemm_rows_experts_bf16(x.data_ptr(), h, wg.data_ptr(), h, act.data_ptr(), I, offs.data_ptr(), E, P, I, h, 1,
                                           0, 0, 0.0, 0.0, rw.data_ptr() if weighted else None,
                                           order.data_ptr() if weighted else None, st), "experts")
    at = 0
    for e, n in enumerate(counts):
        y = x[at:at + n].double() @ wg[e].double().T * (rw[order[at:at + n].long()].double()[:, None] if weighted else 1.0)
        want = _act64(y[:, :I], y[:, I:], "silu")
        assert (act[at:at + n].double() - want).norm() <= 2.5e-3 * want.norm()
        at += n
    assert act[at:].isnan().all()
    act[at:] = 0
    for dtype, bound in ((torch.bfloat16, 2.5e-3), (torch.float32, 1e-6)):
        out = torch.full((P, h), float("nan"), device=DEV, dtype=dtype)
        L.check(lib.slb_gemm_rows_experts_bf16(act.data_ptr(), I, wd.data_ptr(), I, out.data_ptr(), h, offs.data_ptr(), E, P, h,
                                               I, 0, int(dtype == torch.float32), 0, 0.0, 0.0, None, None, st), "experts")
        at = 0
        for e, n in enumerate(counts):
            want = act[at:at + n].double() @ wd[e].double().T
            assert (out[at:at + n].double() - want).norm() <= bound * want.norm()
            at += n
        assert out[at:].isnan().all()
    assert K().gemm_rows_status() == 0


@pytest.mark.parametrize("T,E,top,h,I,half", [(70, 8, 4, 1024, 512, False), (300, 8, 4, 1024, 2048, True), (3, 4, 2, 2048, 1024, False)])
def test_routed_experts_on_sorted_rows(T, E, top, h, I, half):
    """The whole sum, rows read from a wider matrix, with shared rows: against 64 bits with the activation and the result
    rounded (and an expert's rows, in large steps): 6e-3 of the norm."""
    g = gen(T)
    x = torch.randn(T, h + 8, device=DEV, generator=g).bfloat16()[:, 8:]
    wg, wd = ((torch.randn(*s, device=DEV, generator=g) * s[-1] ** -0.5).bfloat16() for s in ((E, 2 * I, h), (E, h, I)))
    ids = torch.stack([torch.randperm(E, device=DEV, generator=g)[:top] for _ in range(T)]).int().contiguous()
    w, shared = torch.rand(T, top, device=DEV, generator=g), torch.randn(T, h, device=DEV, generator=g).bfloat16()
    assert K().moe_tcgen05_pays(h * I) and half == (T * top >= K().moe_vendor_min_pairs)
    got = K().moe_experts(x, ids, w, wg, wd, shared).double()
    want = shared.double()
    for e in range(E):
        t, k = torch.where(ids == e)
        y = x[t].double() @ wg[e].double().T
        want = want.index_add(0, t, w[t, k].double()[:, None] * (_act64(y[:, :I], y[:, I:], "silu") @ wd[e].double().T))
    assert (got - want).norm() <= 6e-3 * want.norm() and K().gemm_rows_status() == 0


def test_rows_of_an_expert_are_rounded_only_where_the_library_rounds_them(monkeypatch):
    """Large steps of large experts with the library's grouped product switched off, and a result of 2,044 columns, which it
    does not take: the experts' rows are float32 until a token's sum, as they are in the other products."""
    g = gen(9)
    T, E, top, h, I = 512, 4, 2, 1024, 2048
    x = torch.randn(T, h, device=DEV, generator=g).bfloat16()
    wg = (torch.randn(E, 2 * I, h, device=DEV, generator=g) * h ** -0.5).bfloat16()
    ids = torch.stack([torch.randperm(E, device=DEV, generator=g)[:top] for _ in range(T)]).int().contiguous()
    w, asked = torch.rand(T, top, device=DEV, generator=g), []
    from servelab_b200.ops import library as L
    lib = L.core()
    real = lib.slb_gemm_rows_experts_bf16
    monkeypatch.setattr(lib, "slb_gemm_rows_experts_bf16", lambda *a: asked.append(a[11:13]) or real(*a))
    for grouped, n_out, f32 in ((True, 1024, 0), (False, 1024, 1), (True, 1020, 1)):
        wd = (torch.randn(E, n_out, I, device=DEV, generator=g) * I ** -0.5).bfloat16()
        monkeypatch.setattr(K(), "moe_vendor_grouped", grouped)
        asked.clear()
        K().moe_experts(x, ids, w, wg, wd, None)
        assert asked == [(1, 0), (0, f32)]


@pytest.mark.parametrize("E,h,I,top", [(16, 1024, 512, 2), (64, 1024, 512, 8), (16, 1024, 768, 4), (8, 1024, 1024, 4), (8, 512, 256, 2)])
def test_a_token_of_routed_experts_does_not_hang_on_the_step(E, h, I, top):
    """Experts below the library's sizes: a token's result is the same bits alone, among a few and in a large step."""
    g, T = gen(E + I), 400
    wg, wd = ((torch.randn(*s, device=DEV, generator=g) * s[-1] ** -0.5).bfloat16() for s in ((E, 2 * I, h), (E, h, I)))
    x, w = torch.randn(T, h, device=DEV, generator=g).bfloat16(), torch.rand(T, top, device=DEV, generator=g)
    ids = torch.stack([torch.randperm(E, device=DEV, generator=g)[:top] for _ in range(T)]).int().contiguous()
    whole = K().moe_experts(x, ids, w, wg, wd, None)
    for n in (1, 3, 17, 64, 150):
        assert torch.equal(K().moe_experts(x[:n], ids[:n], w[:n], wg, wd, None), whole[:n])


@pytest.mark.parametrize("h,I", [(256, 128), (1024, 512), (1024, 2048)])
def test_profiles_name_the_experts_products_alike_in_every_form(h, I):
    """The comparisons of architectures look the two products up by these names, whichever kernels run."""
    from servelab_b200.ops.profile import StepProfile
    g, E, T, top = gen(h), 4, 20, 2
    wg, wd = ((torch.randn(*s, device=DEV, generator=g) * s[-1] ** -0.5).bfloat16() for s in ((E, 2 * I, h), (E, h, I)))
    ids = torch.stack([torch.randperm(E, device=DEV, generator=g)[:top] for _ in range(T)]).int().contiguous()
    with StepProfile() as seen:
        K().moe_experts(torch.randn(T, h, device=DEV, generator=g).bfloat16(), ids, torch.rand(T, top, device=DEV, generator=g), wg, wd, None)
    assert {"moe_plan", "moe_gate_up", "moe_down", "moe_combine"} <= set(seen.totals())


@pytest.mark.parametrize("E,groups,keep,top", [(1, 1, 1, 1), (5, 1, 1, 5), (32, 4, 2, 4), (60, 3, 2, 6), (100, 1, 1, 32), (128, 32, 9, 8),
                                               (128, 2, 1, 3)])
@pytest.mark.parametrize("score_fn", ["softmax", "sigmoid"])
@pytest.mark.parametrize("corrected", [False, True])
def test_choice_of_up_to_128_experts(E, groups, keep, top, score_fn, corrected):
    """Rows with equal scores, zeros of both signs, infinities and no numbers, chosen one by one on the host: the same ids
    (a near tie of choice scores that are not equal by their inputs may fall either way: 2e-6, a few units of the last place
    of a sigmoid, a softmax or their sum with the offset), weights to the rounding of the exponentials and of a sum of 128
    (2e-6)."""
    T, g, near = 41, gen(E + top), 2e-6
    z = (torch.randn(T, E, device=DEV, generator=g) * 2).round(decimals=1)
    z[1] = 0.0
    z[2, ::2] = -0.0
    z[3, E // 2:] = float("-inf")
    if score_fn == "sigmoid":                                  # (a row's softmax has no number once one logit has none)
        z[4, ::3] = float("nan")
        z[5, ::2] = float("inf")
    corr = (torch.randn(E, device=DEV, generator=g) * 0.1).round(decimals=1) if corrected else None
    ids, w = K().moe_route_scored(z, groups, keep, top, 1.5, True, score_fn, corr, 1, 1e-9)
    zc, off, per = z.cpu(), corr.cpu() if corrected else torch.zeros(E), E // groups
    by_logit = score_fn == "sigmoid" and groups == 1 and not corrected
    for t in range(T):
        s = torch.softmax(zc[t], 0) if score_fn == "softmax" else torch.sigmoid(zc[t])
        cs = (zc[t] if by_logit else s + off).tolist()
        score = [max([v for v in cs[k * per:(k + 1) * per] if v == v], default=0.0) for k in range(groups)]
        kept = sorted(range(groups), key=lambda k: (-score[k], k))[:keep]
        least = min(score[k] for k in kept)
        left = [e for e in range(E) if e // per in kept and cs[e] > float("-inf")]
        order = sorted(left, key=lambda e: (-cs[e], e))[:top]
        order += [None] * (top - len(order))
        got = ids[t].tolist()
        chosen = [e for e, want in zip(got, order) if want is not None]
        assert len(set(chosen)) == len(chosen)
        for e, want in zip(got, order):
            if want is None:
                assert e == 0, (t, got, order)
            elif e != want:
                assert (zc[t, e], off[e]) != (zc[t, want], off[want]) and abs(cs[e] - cs[want]) <= near, (t, got, order)
                assert e // per in kept or score[e // per] >= least - near, (t, got, kept)
        if score_fn == "softmax" or t != 4:
            weight = [0.0 if e is None else float(s[i]) for e, i in zip(order, got)]
            want = torch.tensor(weight) / (sum(weight) + 1e-9) * 1.5
            assert torch.allclose(w[t].cpu(), want, rtol=2e-6, atol=1e-7), t


@pytest.mark.parametrize("E,top", [(7, 3), (32, 4), (64, 8), (128, 32)])
@pytest.mark.parametrize("score_fn", ["softmax", "sigmoid"])
def test_choice_of_few_experts_equals_the_general_kernel(E, top, score_fn):
    """The same logits padded with minus infinities to more experts than the other kernel takes: the same bits."""
    z = torch.randn(300, E, device=DEV, generator=gen(E))
    z[7] = z[7, 0]
    wide = torch.full((300, 200), float("-inf"), device=DEV)
    wide[:, :E] = z
    a, b = (K().moe_route_scored(v, 1, 1, top, 2.0, False, score_fn) for v in (z, wide))
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
