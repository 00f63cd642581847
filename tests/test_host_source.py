"""CPU checks of the host sources for state that several threads share: a graph
serves one thread at a time, but threads with graphs of their own (a server's
worker among them) run the same host code together."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCES = sorted(glob.glob(os.path.join(ROOT, "c-saw_b200", "csrc", "*.cu*")))

SAFE = r"(?:const\b|constexpr\b|thread_local\b|std::atomic\b|std::mutex\b|std::once_flag\b|__device__\b|__global__\b|inline\b)"


def test_function_statics_are_safe_between_threads():
    """A variable of static duration inside a function is constant, atomic or
    the thread's own."""
    assert SOURCES
    found = []
    for path in SOURCES:
        for n, line in enumerate(open(path).read().splitlines(), 1):
            if re.match(r"\s+static\s+(?!" + SAFE + r")[^(]*[={;]", line):
                found.append((os.path.basename(path), n, line.strip()))
    assert not found, found


def test_globals_are_safe_between_threads():
    """So is a variable at namespace scope (named g_...)."""
    found, seen = [], 0
    for path in SOURCES:
        for n, line in enumerate(open(path).read().splitlines(), 1):
            m = re.match(r"(?:static\s+)?(?P<type>[A-Za-z_][\w:<>, ]*?)\s+g_\w+\s*(?:[={;\[])", line)
            if m:
                seen += 1
                if not re.match(SAFE, m["type"]):
                    found.append((os.path.basename(path), n, line.strip()))
    assert seen and not found, found


def test_shared_memory_limits_do_not_depend_on_the_call():
    """A kernel's limit of dynamic shared memory holds for the whole process,
    so it is set to one constant and never to what one call needs."""
    seen = 0
    for path in SOURCES:
        for value in re.findall(r"MaxDynamicSharedMemorySize,\s*([^;]*?)\)\)?;", open(path).read()):
            seen += 1
            assert re.fullmatch(r"[A-Z][A-Z0-9_]*|\d+( << \d+)?", value.strip()), (os.path.basename(path), value)
    assert seen
