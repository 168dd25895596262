"""Builds the library's kernels for the host over emu/cuda_emu.h, for tests of their ordering on the CPU.

The sources are used as they stand, with three changes made to a copy: the functions written in PTX are
left out (the header has them), dynamic shared memory becomes a pointer, and kernel launches are taken out of
the launchers (a test's main program runs the kernels itself)."""
import os
import re
import shutil
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
PTX = ("dmma884", "cp_async16", "cp_async8", "cp_async_commit", "cp_async_wait_all", "rcp_approx", "rsqrt_approx",
       "bar_sync", "bar_arrive")


def _drop_function(src, name):
    m = re.search(r"(template <[^>]*>\n)?__device__ __forceinline__ \w+ %s\(" % name, src)
    if not m:
        return src
    at = src.index("{", m.end())
    depth = 0
    while True:
        depth += {"{": 1, "}": -1}.get(src[at], 0)
        at += 1
        if depth == 0:
            return src[:m.start()] + src[at:]


def host_source(src):
    for name in PTX:
        src = _drop_function(src, name)
    src = re.sub(r'asm volatile\("cp\.async\.wait_group.*?"memory"\);', "cp_async_wait_all();", src, flags=re.S)
    src = re.sub(r"extern __shared__ (?:__align__\(16\) )?([\w ]+?) (\w+)\[\];",
                 r"\1* \2 = reinterpret_cast<\1*>(emu::dyn_smem());", src)
    return re.sub(r"\b\w+(?:<[\w, ]*>)?<<<.*?;", ";", src, flags=re.S)


def build(tmp, main, csrc=os.path.join(ROOT, "adaptive_tlr_pilots_b200", "csrc")):
    """The program `main` (C++ that includes the .cu files it runs), compiled; returns its path."""
    tmp = str(tmp)
    inc = os.path.join(tmp, "include")
    dst = os.path.join(tmp, "pkg", "csrc")
    if not os.path.isdir(dst):
        shutil.copytree(os.path.join(ROOT, "include"), inc)
        os.makedirs(dst)
        for f in os.listdir(csrc):
            with open(os.path.join(csrc, f)) as fh:
                text = fh.read()
            with open(os.path.join(dst, f), "w") as fh:
                fh.write(host_source(text))
    path = os.path.join(dst, "main.cpp")
    with open(path, "w") as fh:
        fh.write(main)
    exe = os.path.join(tmp, "main")
    cmd = ["g++", "-std=c++17", "-O1", "-w", "-pthread", "-DTLR_RESTRICT=", "-ffp-contract=off",
           "-I", os.path.join(HERE, "emu"), path, "-o", exe]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-4000:]
    return exe


def run(exe, *args, timeout=300):
    """Standard output of the program, which ends with status 0."""
    res = subprocess.run([exe, *map(str, args)], capture_output=True, text=True, timeout=timeout)
    assert res.returncode == 0, (res.returncode, res.stdout[-2000:], res.stderr[-2000:])
    return res.stdout
