"""Rules of the launches that the kernels' sources have to keep and that no run shows broken.

Kernels that are set up while the kernel before them runs (`launch_after`) wait before their first access, and load nothing through the
read-only path or by an intrinsic with a cache hint, which the compiler may move above that wait.  Grids are sized by the number of SMs that
the device has, not by one written out."""
import glob
import os
import re

from tests.conftest import ROOT

CSRC = os.path.join(ROOT, "raygaussx_b200", "csrc")
DEFINITION = r"(%s)([^;{}]*?)\b(\w+)\(((?:[^(){};]|\([^()]*\))*)\)\s*(?:const\s*)?\{"


def functions(begin=r"__(?:global|device)__"):
    """name -> (kernel?, parameters, body) of every function declared so; bodies of one name in several places are joined."""
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)
        for m in re.finditer(DEFINITION % begin, text):
            depth, end = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            kernel, params, body = out.get(m.group(3), (False, "", ""))
            out[m.group(3)] = (kernel or m.group(1) == "__global__", params + m.group(4), body + text[m.end():end])
    return out


def launched_early():
    text = "".join(open(p).read() for p in glob.glob(os.path.join(CSRC, "*.cu*")))
    return set(re.findall(r"launch_after\(\(?(\w+_kernel)\b", text))


def test_early_kernels_wait_first():
    found, early = functions(), launched_early()
    assert len(early) > 25
    for name in early:
        kernel, _, body = found[name]
        assert kernel and re.match(r"\s*(after_previous\(\);|if \(LATE\) after_previous_then_next\(\);\s*else after_previous\(\);)", body), name


def test_early_kernels_load_nothing_that_may_be_moved():
    found = functions()
    for name in launched_early():
        todo, seen = [name], set()
        while todo:
            f = todo.pop()
            if f in seen or f not in found:
                continue
            seen.add(f)
            _, params, body = found[f]
            assert "__restrict__" not in params, (name, f)
            assert not re.search(r"__ld\w+\(|\bReadOnly\b|global\.nc\b|asm\s*\(\s*\"ld\b", body), (name, f)
            todo += re.findall(r"\b(\w+)\s*(?:<[^;{}()]*>)?\(", body)


def test_launches_before_a_sort_by_cluster_are_looked_at():
    """cluster_sort clears the error of a cluster that the device does not take; an error from before would go with it."""
    callers = [body for name, (_, _, body) in functions(r"cudaError_t").items() if "cluster_sort(" in body and name != "cluster_sort"]
    assert len(callers) == 2
    for body in callers:
        before = body[:body.index("cluster_sort(")]
        assert len(re.findall(r"\blaunch_after\(", before)) == len(re.findall(r"\be = launch_after\(", before)) >= 2
        assert len(re.findall(r"if \(e != cudaSuccess\) return e;|\) != cudaSuccess\) return e;", before)) >= 2


def test_only_launched_kernels_are_counted():
    body = functions(r"inline cudaError_t")["launch_after"][2]
    assert body.index("cudaLaunchKernelEx(") < body.index("if (e == cudaSuccess) note_launch();")
    body = functions(r"cudaError_t")["cluster_sort"][2]
    assert re.search(r"cudaLaunchKernelEx\([^;]*== cudaSuccess\) note_launch\(\);", body)


def test_the_number_of_sms_is_asked_for():
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        text = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)
        assert not re.search(r"\b(148|296|592|1184|9472)\b", text), path
