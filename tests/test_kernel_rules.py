"""Rules of the kernels' sources that a run on a GPU cannot show to be broken (a race that is rarely lost), checked on the text."""
import os
import re

import pytest

_CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "katago_b200", "csrc")


def _kernels():
    """(name, parameter list, body) of every __global__ function."""
    found = []
    for f in sorted(os.listdir(_CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(_CSRC, f)).read())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(text[i], 0)
                i += 1
            params = text[m.end():i - 1]
            start = text.index("{", i)
            depth, j = 1, start + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[j], 0)
                j += 1
            found.append((m.group(1), params, text[start:j]))
    return found


KERNELS = _kernels()


def test_the_sources_are_read():
    names = [k[0] for k in KERNELS]
    assert len(names) >= 30 and {"convTcKernel", "convSmallKernel", "convChainKernel", "gpoolMidKernel"} <= set(names)


@pytest.mark.parametrize("name", [n for n, _, b in KERNELS if "tmemAlloc" in b and "gridDepLaunch" in b])
def test_dependents_start_after_the_tensor_memory_is_allocated(name):
    """A tcgen05 allocation blocks without a limit; a dependent kernel that got onto the SM first could hold the columns it
    waits for while itself waiting for this kernel."""
    body = next(b for n, _, b in KERNELS if n == name)
    last_alloc = max(m.start() for m in re.finditer(r"tmemAlloc(?:Pair)?\(", body))
    launch = [m.start() for m in re.finditer(r"gridDepLaunch\(\)", body)]
    assert len(launch) == 1
    assert "__syncthreads();" in body[last_alloc:launch[0]]


@pytest.mark.parametrize("name", [n for n, _, b in KERNELS if "gridDepWait" in b])
def test_early_kernels_promise_constant_data_for_weights_only(name):
    """const __restrict__ allows loads that are not coherent with, or not ordered after, what the kernel before still writes."""
    params = next(p for n, p, _ in KERNELS if n == name)
    constant = set(re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", params))
    assert constant <= {"w", "wT", "scale", "bias", "layers"}


@pytest.mark.parametrize("name", [n for n, _, b in KERNELS if "mbarWaitWarp" in b])
def test_nothing_is_issued_behind_a_wait_that_ran_out(name):
    """A slot whose wait ran out may still be armed: arming it again in the same phase is past what its barrier can count.  Every
    arming behind a wait therefore asks whether the waits have been met."""
    body = next(b for n, _, b in KERNELS if n == name)
    body = body.split("else if(warp == 1)")[0]  # the feeding warp's part
    issues = list(re.finditer(r"if\((?:one|electOne)\(\)([^{;]*)", body))
    for w in re.finditer(r"\bwait\(&|mbarWaitWarp\(smemU32\(&", body):
        behind = next((i for i in issues if i.start() > w.start()), None)
        assert behind is not None and re.match(r" && (?:go\(\)|live|!\*abortFlag)\)", behind.group(1)), body[w.start():w.start() + 200]


LEAVING = [n for n, _, b in KERNELS if "mbarWaitThread" in b and n != "waitTimeoutSelfTestKernel"]


def test_the_kernels_whose_roles_run_in_one_thread_are_found():
    assert set(LEAVING) == {"convTcKernel", "convSmallKernel"}


@pytest.mark.parametrize("name", LEAVING)
def test_a_thread_leaves_its_role_behind_a_wait_that_ran_out(name):
    """The same for a role inside one thread (mbarWaitThread): whatever follows a wait that failed is left, out of its loops."""
    body = next(b for n, _, b in KERNELS if n == name)
    waits = [m.start() for m in re.finditer(r"(?<!auto )\bwait\((?!\[)", body)]
    assert len(waits) >= 5
    for w in waits:
        line = body[body.rindex("\n", 0, w) + 1:body.index("\n", w)]
        before, behind = body[:w].splitlines()[-1], body[w:].split("\n", 1)[0]
        assert re.search(r"if\((?:[^;{}]* (?:&&|\|\|) )?!$", before), line
        assert re.search(r"\)\) (?:goto \w+;|return;|return false;|\{ ok = false; break; \})$", behind.rstrip()), line
    # a `break` ends one loop; its header, and those around it, ask for `ok`
    for m in re.finditer(r"\{ ok = false; break; \}", body):
        depth, loops = 0, []
        for i in range(m.start() - 1, -1, -1):
            depth += {"}": 1, "{": -1}.get(body[i], 0)
            if depth < 0:
                depth = 0
                header = body[body.rindex("\n", 0, i) + 1:i]
                if "for(" not in header:
                    break
                loops.append(header)
        assert loops and all(re.search(r"&& ok;", h) for h in loops), loops
