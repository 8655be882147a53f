"""Builds the CUDA sources for the CPU (emu/emu.h) and runs them in a child
process, for tests of what must not be tried on a GPU first: index arithmetic,
bounds and wait protocols."""
import functools
import os
import re
import subprocess
import tempfile

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "mce-gpu_b200", "csrc")
_DIR = tempfile.TemporaryDirectory(prefix="mce_emu_")
_LAUNCH = re.compile(r"([A-Za-z_]\w*(?:<[^<>;]*>)?)<<<(.*?)>>>\(([^;]*)\);", re.S)
_DYNAMIC = re.compile(r"extern __shared__ (?:__align__\(\d+\) )?([\w ]+?) (\w+)\[\];")


def _common(text):
    """common.cuh without its PTX: the status bits, and plain loads and stores."""
    bits = "\n".join(re.findall(r"^#define MCE_ERR_.*$|^#define MCE_FULL.*$", text, re.M))
    return f"""#pragma once
#include "emu.h"
#include "{os.path.join(os.path.dirname(HERE), 'include', 'mce.h')}"
{bits}
#define MCE_CUDA(call) do {{ if ((call) != cudaSuccess) return MCE_ECUDA; }} while (0)
namespace mce {{
inline uint64_t globaltimer_ns() {{ static uint64_t t = 0; return t += 1000; }}
inline uint32_t lane_id() {{ return threadIdx.x & 31u; }}
inline uint32_t ld_acquire(const uint32_t *p) {{ return *p; }}
inline void st_release(uint32_t *p, uint32_t v) {{ *p = v; }}
inline void red_release(uint32_t *p, uint32_t v) {{ *p += v; }}
inline uint32_t ld_volatile(const uint32_t *p) {{ return *p; }}
inline unsigned long long ld_volatile(const unsigned long long *p) {{ return *p; }}
inline void mbar_init(unsigned long long *, uint32_t) {{}}
inline void fence_proxy_async_smem() {{}}
inline void mbar_arrive_expect_tx(unsigned long long *, uint32_t) {{}}
inline void bulk_copy_g2s(void *, const void *, uint32_t, unsigned long long *) {{}}
inline bool mbar_wait(unsigned long long *, uint32_t, uint32_t *, uint64_t) {{ return true; }}
}}
"""


def _translate(name, text):
    if name == "common.cuh":
        return _common(text)
    text = re.sub(r"#include <(cuda|cooperative_groups|cub)[^>]*>", "", text)
    text = re.sub(r"asm volatile\(.*?\);", "", text, flags=re.S)
    text = _DYNAMIC.sub(r"\1 *\2 = (\1 *)emu::dynamic();", text)
    return _LAUNCH.sub(r"emu::launch(emu::Config(\2), [&] { \1(\3); });", text)


@functools.lru_cache(maxsize=None)
def build(harness):
    """The program of emu/<harness>.cpp with the sources it includes."""
    tmp = os.path.join(_DIR.name, harness + ".src")
    os.mkdir(tmp)
    for f in os.listdir(CSRC):
        with open(os.path.join(CSRC, f)) as src, open(os.path.join(tmp, f), "w") as dst:
            dst.write(_translate(f, src.read()))
    exe = os.path.join(_DIR.name, harness)
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-I", tmp, "-I", os.path.join(HERE, "emu"),
                    os.path.join(HERE, "emu", harness + ".cpp"), "-o", exe], check=True)
    return exe


def run(harness, *args, arrays=(), timeout=300):
    """Runs it with int32 arrays on its standard input, each after its length;
    (exit status, standard output, standard error)."""
    exe = build(harness)
    data = b"".join(np.int64(len(a)).tobytes() + np.ascontiguousarray(a, np.int32).tobytes()
                    for a in arrays)
    p = subprocess.run([exe] + [str(a) for a in args], input=data, capture_output=True,
                       timeout=timeout)
    return p.returncode, p.stdout, p.stderr.decode()
