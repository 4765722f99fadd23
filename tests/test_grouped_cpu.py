"""Host-side logic around the grouped GEMM: the static schedule, the deferred weight-gradient queue
and the segment-wise linear, all without a GPU."""
import ctypes
import os

import pytest
import torch

from lightron_b200.ops import functional as OF, native


def _plan(shapes, sms=148):
    lib = native._load()
    if lib is None:
        pytest.skip("native library not built")
    n = len(shapes)
    IA = ctypes.c_int * n
    M, N, K = IA(*[s[0] for s in shapes]), IA(*[s[1] for s in shapes]), IA(*[s[2] for s in shapes])
    out = (ctypes.c_longlong * 3)()
    assert lib.lb_gemm_grouped_plan(n, M, N, K, sms, out) == 0
    busiest, work, ctas = out[0], out[1], out[2]
    return busiest * ctas / work, ctas


def test_schedule_balances_weight_gradient_with_data_gradient():
    T = 16384
    alone, _ = _plan([(2560, 2048, T)])                      # 160 tiles on 148 SMs: second wave 8 % full
    paired, ctas = _plan([(2560, 2048, T), (T, 2048, 2560)])
    assert alone > 1.8 and paired < 1.06 and ctas == 148
    # the queued weight gradients of a tensor-parallel layer (TP2 shapes of the 1.1B model)
    assert _plan([(2048, 2816, T), (5632, 2048, T)])[0] < 1.15
    assert _plan([(2048, 1024, T), (1280, 2048, T)])[0] < 1.02
    # fewer tiles than SMs: one tile per CTA
    imb, ctas = _plan([(256, 512, 4096)])
    assert ctas == 4 and imb == 1.0


def _ctas_per_tile(shapes, sms=148):
    IA = ctypes.c_int * len(shapes)
    return native._load().lb_gemm_grouped_ctas_per_tile(len(shapes), *(IA(*[s[i] for s in shapes]) for i in range(3)), sms)


def test_plan_is_the_schedule_of_the_chosen_form():
    """One tile's rows decide between a CTA per 128 rows and a pair per 256: the plan counts the one that the list form launches (alone, the
    first two go to the split form, which has no lists; next to two more problems they do not)."""
    lib = native._load()
    if lib is None:
        pytest.skip("native library not built")
    for shapes, cg, ctas in (([(384, 256, 16384)], 2, 4),            # two 256-row tiles (the second half empty), not three of 128
                             ([(384, 256, 512)], 1, 3),              # a short launch: CTAs
                             ([(16384, 2048, 2048)], 2, 148)):
        IA = ctypes.c_int * 1
        out = (ctypes.c_longlong * 3)()
        assert lib.lb_gemm_grouped_plan(1, *(IA(v) for v in shapes[0]), 148, out) == 0
        kb = shapes[0][2] // 64 + 6
        tiles = -(-shapes[0][0] // (128 * cg)) * -(-shapes[0][1] // 256)
        assert _ctas_per_tile(shapes) == cg and out[2] == ctas and out[1] == cg * tiles * kb, shapes
        assert out[0] == -(-tiles // (ctas // cg)) * kb
    assert _ctas_per_tile([(0, 8, 8)]) < 0


@pytest.mark.parametrize("shapes,cg", [
    # the store of a tile outlasts its main loop: pairs were 4 to 24 % slower, whatever the number of tiles
    ([(16384, 4096, 256)], 1), ([(8192, 5632, 512)], 1), ([(16384, 2304, 768)], 1), ([(4096, 4096, 768)], 1),
    # it does not: 4 to 11 % faster
    ([(8192, 4096, 1024)], 2), ([(4096, 4096, 1536)], 2), ([(16384, 768, 1536)], 2), ([(16384, 5632, 4096)], 2),
    # one or two short tiles per SM: the setup (the last one goes to the split form unless a third problem comes with it)
    ([(1000, 2304, 768)], 1), ([(4096, 2304, 768)], 1), ([(2048, 2304, 2048)], 1), ([(512, 768, 768), (512, 768, 768)], 1),
    # the weight gradient's long tiles carry the data gradient's short ones
    ([(2304, 768, 8192), (8192, 768, 2304)], 2),
])
def test_pairs_are_chosen_where_they_are_faster(shapes, cg):
    if native._load() is None:
        pytest.skip("native library not built")
    assert _ctas_per_tile(shapes) == cg


@pytest.mark.parametrize("shapes,parts", [
    ([(128, 768, 2048)], 4), ([(128, 2048, 5632)], 4), ([(128, 2304, 768)], 1), ([(16, 11264, 2048)], 1), ([(8, 8, 8)], 1),
    ([(768, 768, 1000), (1000, 768, 768)], 1), ([(1000, 768, 2048)], 2),
    # enough tiles of 128 x 256 to fill the chip, or more than two problems
    ([(16384, 2048, 2048)], 0), ([(1000, 4096, 768)], 0), ([(1000, 32000, 768)], 0), ([(2048, 2048, 2048)], 0), ([(128, 768, 2048)] * 3, 0),
])
def test_short_launches_are_split(shapes, parts):
    lib = native._load()
    if lib is None:
        pytest.skip("native library not built")
    IA = ctypes.c_int * len(shapes)
    assert lib.lb_gemm_grouped_parts(len(shapes), *(IA(*[s[i] for s in shapes]) for i in range(3)), 148) == parts


def test_schedule_rejects_bad_arguments():
    lib = native._load()
    if lib is None:
        pytest.skip("native library not built")
    IA = ctypes.c_int * 1
    out = (ctypes.c_longlong * 3)()
    assert lib.lb_gemm_grouped_plan(1, IA(0), IA(8), IA(8), 148, out) != 0
    assert lib.lb_gemm_grouped_plan(9, IA(8), IA(8), IA(8), 148, out) != 0


def test_attention_backward_refuses_a_short_workspace():
    """The size travels with the pointer: a workspace that is too small is refused before anything is launched."""
    lib = native._load()
    if lib is None:
        pytest.skip("native library not built")
    need = lib.lb_flash_bwd_ws_bytes(2, 129, 3, 64)
    assert need == 2 * 3 * 256 * (2 + 64) * 4 and lib.lb_flash_bwd_ws_bytes(1, 8, 1, 32) == 0
    assert lib.lb_flash_bwd_ws_bytes(8, 1 << 20, 64, 128) == 8 * 64 * (1 << 20) * 130 * 4          # past 32 bits
    strides = [192] * 8
    assert lib.lb_flash_bwd_tc_ws(*[0] * 7, need - 1, 0, 0, 0, 2, 129, 129, 3, 3, 64, *strides, 1.0, 1, 0) == -6
    assert lib.lb_flash_bwd_cp_ws(*[0] * 7, need - 1, 0, 0, 0, 2, 129, 129, 200, 3, 3, 64, *strides, 1.0, 1, 0) == -6
    assert lib.lb_flash_bwd_cp_ws(*[0] * 7, need, 0, 0, 0, 2, 129, 129, 100, 3, 3, 64, *strides, 1.0, 1, 0) == -3


def _fake_gemm_grouped(problems):
    outs = []
    for a, b, a_mn, b_mn, out, acc in problems:
        A = a.t() if a_mn else a
        Bm = b if b_mn else b.t()
        r = A.float() @ Bm.float()
        if out is None:
            out = torch.empty(r.shape, dtype=a.dtype)
        out.copy_((out.float() + r if acc else r).to(out.dtype))
        outs.append(out)
    return outs


class _DeferringLinear(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w):
        ctx.save_for_backward(x, w)
        ctx.params = (w,)
        return x @ w.t()

    @staticmethod
    def backward(ctx, dy):
        x, w = ctx.saved_tensors
        assert OF.direct_wgrad_ok(ctx.params)
        OF.defer_wgrad(dy.contiguous(), x, ctx.params)
        return dy @ w, None


def test_deferred_weight_gradients_flush_once_at_end_of_backward(monkeypatch):
    monkeypatch.setattr(OF, "gemm_grouped", _fake_gemm_grouped)
    launches = []
    real = OF.gemm_grouped
    monkeypatch.setattr(OF, "gemm_grouped", lambda probs: (launches.append(len(probs)), real(probs))[1])
    torch.manual_seed(0)
    arena = torch.zeros(3 * 16 * 16)
    ws, fired = [], []
    for i in range(3):
        w = torch.nn.Parameter(torch.randn(16, 16) * 0.3)
        w.grad = arena[i * 256:(i + 1) * 256].view(16, 16)
        w._lb_direct_grad = True
        w._lb_grad_hooks = (lambda p, i=i: fired.append((i, bool(getattr(p, "_lb_wgrad_pending", False)))),)
        ws.append(w)
    x = torch.randn(5, 16, requires_grad=True)
    h = x
    for w in ws:                                        # every weight is used twice per forward
        h = _DeferringLinear.apply(h, w) + 0.5 * _DeferringLinear.apply(h, w)
    h.sum().backward()
    assert launches == [6]                              # six queued products, one grouped launch
    assert sorted(i for i, _ in fired) == [0, 0, 1, 1, 2, 2] and not any(p for _, p in fired)
    assert not OF._WQ and all(not w._lb_wgrad_pending for w in ws)
    ws2 = [w.detach().clone().requires_grad_(True) for w in ws]
    x2 = x.detach().clone().requires_grad_(True)
    h2 = x2
    for w in ws2:
        h2 = h2 @ w.t() + 0.5 * (h2 @ w.t())
    h2.sum().backward()
    for w, w2 in zip(ws, ws2):
        assert torch.allclose(w.grad, w2.grad, atol=1e-4, rtol=1e-4)
    assert torch.allclose(x.grad, x2.grad, atol=1e-4, rtol=1e-4)


def test_grouped_linear_segments_match_per_segment_math():
    torch.manual_seed(1)
    x = torch.randn(11, 16, requires_grad=True)
    groups = [(torch.randn(8, 16, requires_grad=True), torch.randn(8, 16, requires_grad=True)) for _ in range(3)]
    counts = [4, 0, 5]                                  # two rows are beyond every segment
    y = OF.grouped_linear(x, counts, groups)
    assert y.shape == (11, 16) and y[9:].abs().max().item() == 0
    want0 = torch.cat([x[:4] @ groups[0][0].t(), x[:4] @ groups[0][1].t()], dim=1)
    want2 = torch.cat([x[4:9] @ groups[2][0].t(), x[4:9] @ groups[2][1].t()], dim=1)
    assert torch.allclose(y[:4], want0, atol=1e-5) and torch.allclose(y[4:9], want2, atol=1e-5)
    y.square().sum().backward()
    assert groups[1][0].grad is None or groups[1][0].grad.abs().max().item() == 0
    assert x.grad[9:].abs().max().item() == 0 and x.grad[:9].abs().max().item() > 0


def test_bucket_hook_counts_each_parameter_once_and_skips_pending_or_unsynced():
    from lightron_b200 import mesh
    from lightron_b200.config import ModelArgs
    from lightron_b200.models import LightronTransformer, init_weights
    from lightron_b200.optim import DistributedAdamW
    mesh.set_context(None)
    args = ModelArgs(dim=32, n_layers=1, n_heads=2, n_kv_heads=2, vocab_size=64, intermediate_size=64, max_seq_len=16)
    m = LightronTransformer(args, dtype=torch.float32, device=torch.device("cpu"))
    init_weights(m, 0)
    opt = DistributedAdamW(m, lr=1e-3)
    assert opt.grad_shard.data_ptr() == opt.flat_grads.data_ptr()        # no replicas: shards alias the arenas
    b = opt.buckets[0]
    launched = []
    opt._launch_reduce = lambda bb, async_op: launched.append(bb)
    hook = opt._make_hook(b)
    p0, p1 = opt.params[0], opt.params[1]
    b.pending, b.seen = 2, set()
    hook(p0); hook(p0)                                   # by hand and again by autograd: one count
    assert b.pending == 1 and not launched
    p1._lb_wgrad_pending = True
    hook(p1)                                             # its weight gradient is still queued
    assert b.pending == 1
    p1._lb_wgrad_pending = False
    with opt.no_sync():
        hook(p1)                                         # micro-batch without gradient sync
    assert b.pending == 1
    hook(p1)
    assert b.pending == 0 and launched == [b]
    opt._reset_buckets()
    assert b.pending == b.n_params and not b.seen


_SAN_SCRIPT = r'''
import ctypes, random, sys
lib = ctypes.CDLL(sys.argv[1])
random.seed(0)
# host-only entry points (no CUDA call): the static schedule of the grouped GEMM for many shape sets
for trial in range(200):
    n = random.randint(1, 8)
    IA = ctypes.c_int * n
    M = IA(*[random.choice([8, 128, 1000, 4096, 16384]) for _ in range(n)])
    N = IA(*[random.choice([8, 264, 2048, 11264]) for _ in range(n)])
    K = IA(*[random.choice([8, 200, 2048, 16384]) for _ in range(n)])
    out = (ctypes.c_longlong * 3)()
    rc = lib.lb_gemm_grouped_plan(n, M, N, K, random.choice([1, 7, 148]), out)
    assert rc == 0 and out[0] > 0 and out[1] >= out[0] and out[2] >= 1, (rc, list(out))
IA1 = ctypes.c_int * 1
out = (ctypes.c_longlong * 3)()
assert lib.lb_gemm_grouped_plan(0, IA1(8), IA1(8), IA1(8), 148, out) != 0
assert lib.lb_gemm_grouped_plan(1, IA1(-5), IA1(8), IA1(8), 148, out) != 0
lib.lb_set_flag_wait_ns.argtypes = [ctypes.c_ulonglong]
assert lib.lb_set_flag_wait_ns(5_000_000) == 0
assert lib.lb_gemm_grouped_cached() == 0
print("SANITIZED_HOST_OK")
'''


def test_host_code_under_address_and_ub_sanitizers(tmp_path):
    """The C++ host side of the library (argument checks, the grouped GEMM's schedule builder) built with
    -fsanitize=address,undefined and driven without a GPU: any out-of-bounds access, use after free or
    undefined arithmetic in it aborts the child process."""
    import shutil
    import subprocess
    import sys
    from lightron_b200.csrc import build as B
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    if not os.path.exists(nvcc) or shutil.which("gcc") is None:
        pytest.skip("needs nvcc and gcc")
    asan = subprocess.run(["gcc", "-print-file-name=libasan.so"], capture_output=True, text=True).stdout.strip()
    if not os.path.isabs(asan) or not os.path.exists(asan):
        pytest.skip("libasan not installed")
    lib = B.build_sanitized(str(tmp_path / "liblightron_b200_asan.so"))
    script = tmp_path / "san.py"
    script.write_text(_SAN_SCRIPT)
    env = dict(os.environ, LD_PRELOAD=asan, ASAN_OPTIONS="detect_leaks=0:protect_shadow_gap=0:abort_on_error=1",
               UBSAN_OPTIONS="halt_on_error=1:print_stacktrace=1")
    r = subprocess.run([sys.executable, str(script), lib], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "SANITIZED_HOST_OK" in r.stdout, r.stdout[-1500:] + r.stderr[-3000:]


def test_host_module_of_another_torch_is_not_loaded(monkeypatch):
    """The module of the autograd nodes names the torch it was built against: for another one it is rebuilt, and never loaded."""
    from lightron_b200.csrc import build
    if not os.path.exists(build.HOST_LIB):
        pytest.skip("native library not built")
    assert build.host_built_for_this_torch()
    monkeypatch.setattr(torch, "__version__", torch.__version__ + "x")
    assert build.needs_build() and not build.host_built_for_this_torch()
    with pytest.warns(UserWarning, match="not built for torch"):
        assert native._load_host_ops() is None


def _conditions(src, at):
    """The conditions of the if statements whose braces enclose position ``at`` of ``src``."""
    out, depth = [], 0
    for i in range(at, -1, -1):
        if src[i] == "}":
            depth += 1
        elif src[i] == "{" and depth:
            depth -= 1
        elif src[i] == "{":
            head = src[:i].rstrip()
            if head.endswith(")"):
                n = 0
                for j in range(len(head) - 1, -1, -1):
                    n += (head[j] == ")") - (head[j] == "(")
                    if n == 0:
                        break
                if head[:j].rstrip().split()[-1] in ("if", "constexpr"):
                    out.append(head[j + 1:-1])
    return out


def test_parts_of_a_reduction_are_exchanged_whatever_failed():
    """A CTA of the split GEMM that has given up still sends its parts and waits for those of the others, on words that no abort sets: stores
    into a CTA's shared memory have arrived before it may end.  (Read from the source: no test makes a GPU miss them.)"""
    from lightron_b200.csrc import build
    src = open(os.path.join(build.HERE, "gemm_split.cu")).read()
    src = "\n".join(line.split("//")[0] for line in src.splitlines())
    body = src[src.index("void __launch_bounds__(NUM_THREADS, 2) gemm_split_kernel"):src.index("int launch(const Params& gp")]
    sends, waits = [body.index(t) for t in ("st_cluster_v4(dst, r", "mbar_wait<true>(received")]
    assert _conditions(body, body.index("bw::tmem_ld32(taddr + set * HB, r)"))[0] == "ok"      # (what the search finds where there is one)
    for at in (sends, waits):
        assert sorted(_conditions(body, at)) == ["KS > 1", "warp >= 2"]
    words = body[waits:].split(")")[0].split(",")[-1].strip()
    assert words == "s_sums" and "give_up(s_sums" not in body and body.count(words + "[0] = ") == 1
    assert body.index("mbar_wait<true>(received") < body.index("bw::cluster_wait()")


@pytest.mark.parametrize("epi", [0, 1, 2])
def test_outputs_that_are_missing(epi):
    """Only the SwiGLU forward may leave out C; elsewhere a null C is refused before anything is launched (on a machine without a GPU
    the call that is not refused ends at its first CUDA call)."""
    if torch.cuda.is_available():
        pytest.skip("host checks; the addresses are made up")
    lib = native._load()
    if lib is None:
        pytest.skip("native library not built")
    V, I, L = ctypes.c_void_p * 1, ctypes.c_int * 1, ctypes.c_longlong * 1
    n, half = (512, 256) if epi == 1 else (256, 256)
    for C in (0, 4096):
        head = (1, V(4096), V(4096), V(C), I(256), I(n), I(512), L(512), L(512), L(2 * half), I(0), I(0), I(0), I(epi), V(4096), L(2 * half), I(half))
        refused = [lib.lb_gemm_grouped_epi(*head, None), lib.lb_gemm_split(*head, 1, None),
                   lib.lb_gemm_ragged_epi(4096, V(4096), C, 4096, 1, 256, 0, n, 512, 512, 512, 2 * half, 0, epi, 4096, 2 * half, half, None, 0, None)]
        if epi == 0:
            refused.append(lib.lb_gemm_ragged_wgrad(4096, 4096, V(C), 4096, 1, 256, 0, 256, 512, 256, 512, 512, 0, None))
        assert [r == -1 for r in refused] == [C == 0 and epi != 1] * len(refused), (C, refused)


def test_expert_gemms_are_planned_for_the_rows_that_arrive(monkeypatch):
    """Several ranks' exchange buffers hold twice what an even routing brings (capacity factor 2): the form of the expert GEMMs goes by the latter."""
    from lightron_b200.parallel import ep_fused
    lib = native._load()
    if lib is None:
        pytest.skip("native library not built")
    assert ep_fused.capacity(1000, 2, 1, 8, 2.0) == (2048 + 8 * 128, 2048)
    assert ep_fused.capacity(1000, 2, 4, 2, 2.0) == (4096 + 2 * 128, 2000) and ep_fused.capacity(1000, 2, 4, 2, 0.5) == (1024 + 2 * 128, 1000 + 24)
    T, topk, LE, H = 1024, 2, 8, 2048                    # 256 rows per expert: weight gradients in pairs take 59 us, in single CTAs 48
    cap, rows = ep_fused.capacity(T, topk, 8, LE, 2.0)
    form = lambda held, n, k: lib.lb_gemm_ragged_ctas_per_tile(LE, held, n, k, 148)
    assert form(cap, H, 0) == 2 and form(rows + LE * 128, H, 0) == 1
    seen, calls = [], []
    monkeypatch.setattr(ep_fused, "workspace", lambda *a: None)
    monkeypatch.setattr(ep_fused._FusedMoE, "apply", lambda *a: seen.append(a[2]))
    monkeypatch.setattr(ep_fused.dist, "get_world_size", lambda group: 8)
    ep_fused.fused_moe(torch.zeros(T, H), None, (), 8 * LE, topk, object(), 0)
    assert seen[0]["rows"] == rows == T * topk
    monkeypatch.setattr(native, "call", lambda name, *a: calls.append((name, a)))
    monkeypatch.setattr(native, "stream_ptr", lambda: 0)
    t = torch.zeros(8, 8, dtype=torch.bfloat16)
    ep_fused._ragged(t, [t], t, t, LE, cap, H, 512, False, rows=rows)
    ep_fused._ragged_wgrad(t, t, [t], t, LE, cap, 512, H, False, rows)
    assert [a[4:9] for _, a in calls] == [(LE, cap, rows, H, 512), (LE, cap, rows, 512, H)]
