"""The library's own way in: its list of launchers is that of the sources, and its checks are those of ops._why_not."""
import ctypes
import glob
import os
import re
import subprocess

import pytest
import torch

from air_b200.csrc import build, ops


def prototypes():
    """The kinds of the arguments of every launcher, by its name."""
    found = {}
    for path in glob.glob(os.path.join(build.HERE, "*.cu")):
        with open(path) as f:
            source = f.read()
        for name, arguments in re.findall(r"AIR_API\s+int\s+(air_\w+)\(([^)]*)\)\s*{", source):
            found[name] = ["pointer" if "*" in a or "cudaStream_t" in a else a.rsplit(None, 1)[0].replace("const ", "").strip()
                           for a in arguments.split(",")]
    return found


def test_signatures_are_those_of_the_sources():
    kinds = {ctypes.c_void_p: "pointer", ctypes.c_int: "int", ctypes.c_longlong: "long long", ctypes.c_float: "float"}
    found = prototypes()
    for name, types in ops._SIGNATURES.items():
        assert [kinds[t] for t in types] == found[name], name


def test_functions_that_c_programs_call_keep_their_arguments():
    """Functions with more arguments stand beside the ones that were there, under names of their own."""
    p, i, l, f = "pointer", "int", "long long", "float"
    were = {"air_decode_combine": [p, p, p, p, i, i, i, i, p],
            "air_decode_attention_tma_fresh": [p, i, p, p, i, p, l, p, i, p, p, p, p, p, i, i, i, i, i, i, f, i, p, p],
            "air_expert_stream": [p, i, p, i, i, i, p, p, p, i, i, i, p, i, p, i, l, i, p, f, f, f, i, p, p]}
    found, lib = prototypes(), build.library()
    for name, arguments in were.items():
        assert found[name] == arguments and hasattr(lib, name), name
    assert lib.air_decode_combine(None, None, None, None, 1, 1, 7, 2, None) == 100001


def waits(source):
    """Of every bounded wait on a barrier in memory: its line, what stands ahead of the blocks around it, its statement up to it, and what
    follows the statement."""
    source = re.sub(r"//[^\n]*", "", source)
    around, depth, begin = [], 0, 0
    for m in re.finditer(r"[(){};]|\bmbar_wait\(", source):
        c, at = m.group(), m.start()
        if c == "mbar_wait(":
            yield source.count("\n", 0, at) + 1, [opening for opening, _ in around], source[begin:at], source[source.index(";", at) + 1:].lstrip()
        if c.endswith("("):
            depth += 1
        elif c == ")":
            depth -= 1
        elif c == "{":
            around.append((source[begin:at], depth))
            depth, begin = 0, at + 1
        elif c == "}":
            depth, begin = around.pop()[1], at + 1
        elif depth == 0:
            begin = at + 1


def test_a_warp_goes_on_together_behind_a_wait():
    """A wait that runs out answers each thread by itself.  Products, reads of tensor memory and barriers of a block want whole warps:
    every wait is voted on, or made by one thread, or the warp comes together behind it and nothing is left out by those whose wait ran
    out.  (elementwise.cu: each thread chooses where it reads its own numbers.  attention_prefill_tc.cu: its warps leave thread by thread
    when a wait has run out; a vote, or going on without leaving, costs 3 to 8 % of the kernel.)"""
    one = re.compile(r"(lane|tid|threadIdx\.x) == 0( &&|\))|elect_one\(\)")
    voted, together, alone, left = 0, 0, 0, []
    for path in sorted(glob.glob(os.path.join(build.HERE, "*.cu"))):
        with open(path) as f:
            source = f.read()
        for line, around, statement, behind in waits(source):
            if re.search(r"__all_sync\(0xffffffffu,[^;]*$|__syncthreads_or\(!$", statement):
                voted += 1
            elif re.search(r"\bok = $", statement) and re.match(r"(if \([^{;]*\) \{\s*)?__syncwarp\(\);", behind):
                together += 1
            elif any(one.search(opening) for opening in around + [statement]):
                alone += 1
            elif os.path.basename(path) not in ("elementwise.cu", "attention_prefill_tc.cu"):
                left.append(f"{os.path.basename(path)}:{line}")
    assert not left and voted > 20 and alone > 5, (left, voted, together, alone)


def test_what_the_attention_asks_for_ahead():
    """Up to 24 MB of two tensors in their order; nothing where the first alone is larger, and never beyond a tensor's end."""
    of = lambda mb: torch.empty(mb << 20, dtype=torch.uint8)
    small, half, large = of(8), of(16), of(25)
    assert ops.asked_ahead(()) == [None, 0, None, 0]
    assert ops.asked_ahead((small,)) == [small.data_ptr(), 8 << 20, None, 0]
    assert ops.asked_ahead((small, large)) == [small.data_ptr(), 8 << 20, large.data_ptr(), 16 << 20]
    assert ops.asked_ahead((half, small)) == [half.data_ptr(), 16 << 20, small.data_ptr(), 8 << 20]
    assert ops.asked_ahead((large, small)) == [None, 0, None, 0]
    across = half.view(4, -1).t()
    assert ops.asked_ahead((across, small)) == [across.data_ptr(), 0, small.data_ptr(), 8 << 20]


@pytest.mark.gpu
@pytest.mark.parametrize("D,splits", [(64, 1), (128, 7), (256, 32)])
def test_the_merge_alone(D, splits):
    """air_decode_combine against the same merge in 64 bits; a padding token's row stays as it is."""
    T, H = 3, 5
    g = torch.Generator().manual_seed(D)
    o, m, n = torch.randn(T, H, splits, D, generator=g), torch.randn(T, H, splits, generator=g) * 4, torch.rand(T, H, splits, generator=g) + 1
    ml, slots = torch.stack([m, n], dim=-1).cuda(), torch.tensor([0, -1, 4], dtype=torch.int32, device="cuda")
    out, parts = torch.full((T, H, D), 7.0, dtype=torch.bfloat16, device="cuda"), o.cuda()
    f = build.library().air_decode_combine
    f.argtypes = [ctypes.c_void_p] * 4 + [ctypes.c_int] * 4 + [ctypes.c_void_p]
    assert f(parts.data_ptr(), ml.data_ptr(), slots.data_ptr(), out.data_ptr(), T, H, D, splits, torch.cuda.current_stream().cuda_stream) == 0
    w = torch.exp2(m.double() - m.double().amax(-1, keepdim=True))
    want = (o.double() * w[..., None]).sum(2) / (n.double() * w).sum(-1)[..., None]
    got = out.cpu().double()
    assert (got[1] == 7).all() and ((got - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5)[[0, 2]].all()


def test_the_library_is_one_of_c_functions(tmp_path):
    """A program without Python and torch loads the library and calls a launcher (which refuses the arguments: no device is needed)."""
    source, program = tmp_path / "host.c", str(tmp_path / "host")
    source.write_text("""
#include <dlfcn.h>
#include <stdio.h>
int main(int n, char** a) {
    void* lib = dlopen(a[1], RTLD_NOW);
    if (!lib) return puts(dlerror()), 2;
    int (*f)(const float*, const float*, const float*, float*, int, int, int, int, void*) = dlsym(lib, "air_gemm_f32");
    if (!f) return puts(dlerror()), 3;
    printf("%d %d\\n", f(0, 0, 0, 0, 1, 1, -1, 0, 0), f(0, 0, 0, 0, 0, 1, 1, 0, 0));
    return 0;
}
""")
    subprocess.run(["gcc", str(source), "-o", program, "-ldl"], check=True)
    done = subprocess.run([program, build.build()], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    assert (done.returncode, done.stdout.split()) == (0, ["100001", "0"]), done.stdout


@pytest.mark.gpu
def test_a_tensor_is_checked_as_in_python():
    t = torch.zeros(3, 4, device="cuda")
    fits = [((t, "t"), {}), ((t, "t", (torch.float32,)), {}), ((t, "t", (torch.bfloat16, torch.float32), (3, None)), {}),
            ((t, "t", None, (3, 4)), {}), ((t, "t", None, t.shape), {}), ((t, "t"), {"shape": (3, 4)}),
            ((t[:0], "t", None, (0, 4)), {}), ((t[0, 0], "t", None, ()), {}), ((torch.nn.Parameter(t), "t"), {})]
    for args, names in fits:
        assert ops._req(*args, **names) is args[0] and ops._why_not(*args, **names) is args[0]
    for args, names in [((t.cpu(), "t"), {}), ((t.t(), "t"), {}), ((t, "t", (torch.int32,)), {}), ((t, "t", None, (3, 4, 1)), {}),
                        ((t, "t", None, (4, 4)), {}), ((t, "t"), {"shape": (None, 5)}), ((None, "t"), {}), (([1.0], "t"), {})]:
        said = []
        for check in (ops._req, ops._why_not):
            with pytest.raises(ops.KernelError) as e:
                check(*args, **names)
            said.append(str(e.value))
        assert said[0] == said[1]


def test_new_tensors_of_every_form_that_torch_takes():
    """Sizes as a list, a device by its name: what the library's own function does not read goes to torch (no device is needed)."""
    entry = build.entry()
    entry.set_any_empty(ops._any_empty)
    for shape, device in (((2, 3), "cpu"), ([2, 3], "cpu"), ([4], torch.device("cpu")), ((2, 0), torch.device("cpu")), (5, "cpu")):
        a, b = entry.empty(shape, torch.bfloat16, device), torch.empty(shape, dtype=torch.bfloat16, device=device)
        assert a.shape == b.shape and a.dtype == b.dtype and a.device == b.device
    for wrong in ((), ((2, 3), torch.float32), ((2, 3), 7, "cpu"), ("x", torch.float32, "cpu"), ((2, "x"), torch.float32, torch.device("cpu"))):
        with pytest.raises(TypeError):
            entry.empty(*wrong)


@pytest.mark.gpu
def test_a_runtime_whose_device_is_a_name():
    """Parts of a runtime that was given its device as a text, as torch takes it."""
    from types import SimpleNamespace
    from air_b200.parts.base import Runtime
    from air_b200.parts.embedding import TokenEmbedding
    from air_b200.parts.spec import PartSpec
    table = torch.randn(7, 8, device="cuda").bfloat16()
    part = TokenEmbedding(PartSpec("tokens", {"hidden": 8, "vocab": 7}), "t")
    part.load({"t": table}, Runtime("cuda", torch.bfloat16))
    ctx = SimpleNamespace(num_tokens=2, token_ids=torch.tensor([3, 6], dtype=torch.int32, device="cuda"), status=None, last_token=None)
    (h,) = part.forward(ctx, ())
    assert torch.equal(h, table[[3, 6]].float())


@pytest.mark.gpu
def test_new_tensors_and_launches():
    dev = torch.device("cuda:0")
    ops.empty(1, torch.float32, dev)
    for shape in ((2, 3), (0, 5), (), 7, torch.Size((4,))):
        a, b = ops.empty(shape, torch.bfloat16, dev), torch.empty(shape, dtype=torch.bfloat16, device=dev)
        assert a.shape == b.shape and a.dtype == b.dtype and a.device == b.device and a.is_contiguous()
    with pytest.raises(RuntimeError):
        ops.empty((-1,), torch.float32, dev)
    with pytest.raises(torch.cuda.OutOfMemoryError):
        ops.empty((1 << 45,), torch.float32, dev)
    f = build.entry().air_add_parts
    for wrong in ((), (0,) * 5, (None, None, "x", 0, 0, None), (None, None, 0.5, 0, 0, None)):
        with pytest.raises(TypeError):
            f(*wrong)
    # a launch on the stream that is current
    h, d = torch.zeros(1, 1 << 20, device=dev), torch.ones(1, 1 << 20, device=dev)
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        ops.add_parts(h, d)
    s.synchronize()
    assert float(h.sum()) == 1 << 20
