"""Launches from several host threads. What a kernel may use of shared memory is an attribute of the kernel, not of a launch:
it has to be one value whatever a call's sizes are, or a thread's small call takes it away from another's large one."""
import os
import re
import threading

import pytest
import torch

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llm_infer_engine_b200", "csrc")
DEV = "cuda"
# what the value may be made of: constants of the file or of the kernel's template
CONSTANT = re.compile(r"^(\(int\))?(TB \* )?(k[A-Z]\w*|[A-Z]\w*(<[^>]*>)?::(k[A-Z]\w*|[A-Z]+|smem_bytes\((T::k[A-Z]\w*)?\))"
                      r"|lt_smem_bytes\(k[A-Z]\w*\))$")


@pytest.mark.parametrize("source", sorted(f for f in os.listdir(CSRC) if f.endswith(".cu")))
def test_a_kernels_limit_is_one_value(source):
    with open(os.path.join(CSRC, source)) as f:
        text = " ".join(f.read().replace("\\\n", " ").split())
    for m in re.finditer(r"cudaFuncAttributeMaxDynamicSharedMemorySize, (.*?)\);", text):
        value = m.group(1).strip()
        assert CONSTANT.match(value), f"{source}: {value}"
        name = re.sub(r"^\(int\)", "", value)
        if re.fullmatch(r"k[A-Z]\w*", name):
            assert re.search(r"constexpr (int|size_t) (\w+ = \w+, )*" + name + r"\b", text) or name == "kMostRowSmem", name


def _in_threads(calls, rounds):
    """Runs every function of `calls` `rounds` times in a thread and on a stream of its own; they return a tensor that has
    to come out the same each time."""
    errors, start = [], threading.Barrier(len(calls))

    def work(call):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                want = call().clone()
                start.wait(60)
                got = [call() for _ in range(rounds)]
                torch.cuda.current_stream().synchronize()
                assert all(torch.equal(g, want) for g in got)
        except Exception as e:                                                               # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


@pytest.mark.gpu
@pytest.mark.parametrize("kernel", ["grouped", "route", "latent"])
def test_threads_with_different_sizes(kernel):
    from llm_infer_engine_b200.kernels import ops
    g = torch.Generator().manual_seed(3)
    bf = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16).to(DEV)                    # noqa: E731
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)                             # noqa: E731
    calls = []
    if kernel == "grouped":
        for k in (64, 640):
            a, w = bf(70, 2 * k), bf(2, 96, k)

            def call(a=a, w=w, k=k):
                out = torch.zeros(70, 192, dtype=torch.bfloat16, device=DEV)
                ops.batched_gemm_nt(a, w, out, k, 96, k)
                return out
            calls.append(call)
    elif kernel == "route":
        for d in (6272, 12000):                      # two tokens a block, more than 48 KB
            x, w = bf(300, d), torch.randn(4, d, generator=g).to(DEV)

            def call(x=x, w=w):
                ids, wt = torch.empty(300, 2, dtype=torch.int32, device=DEV), torch.empty(300, 2, device=DEV)
                ops.moe_route(x, w, None, ids, wt)
                return wt
            calls.append(call)
    else:
        for hd, hdv in ((64, 64), (320, 256)):
            q, cache = bf(130, 2 * hd), bf(4, 1, 64, hd)

            def call(q=q, cache=cache, hd=hd, hdv=hdv):
                out = torch.empty(130, 2 * hdv, dtype=torch.bfloat16, device=DEV)
                ops.attention_latent_tc(q, cache, cache[..., :hdv], out, i32([0, 130]), i32([0]), i32([0]), i32([[0, 1, 2]]),
                                        64, 1, 130, 2, hd, 0.1)
                return out
            calls.append(call)
    _in_threads(calls, 1500)
    ops.check_tc_status(torch.device(DEV, 0))
