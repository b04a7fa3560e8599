"""Rules of the host code that need no device: each is a header of plain C++, compiled here."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "macseek_b200", "csrc")


def run_cpp(tmp_path, header, body):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text('#include "%s"\n#include <cstdio>\nusing namespace msb;\nint main() {\n%s\n}\n' % (header, body))
    subprocess.check_call(["g++", "-std=c++17", "-I" + CSRC, str(src), "-o", str(exe)])
    return [tuple(int(v) for v in line.split()) for line in subprocess.check_output([str(exe)], text=True).splitlines()]


def test_hc_step_takes_the_ticket_kernel_where_no_cluster_runs(tmp_path):
    cases = [(4096, 1, 1, 7, 7), (4096, 7, 1, 7, 7), (4096, 8, 1, 7, 7), (4096, 20, 1, 7, 7),     # one token each, then four
             (4096, 1, 1, 0, 0), (4096, 20, 1, 0, 0), (4096, 20, 1, 7, 0), (4096, 1, 1, 1, 0),      # a device that places none (of one form)
             (4096, 1, 0, 7, 7), (512, 1, 1, 0, 0), (6144, 1, 1, 7, 7), (4000, 1, 1, 7, 7)]         # alignment, widths
    got = run_cpp(tmp_path, "hc_route.h", "\n".join(
        'printf("%%d %%d\\n", hc_route(%d, %d, %d, %d, %d).tokens, hc_route(%d, %d, %d, %d, %d).clusters);' % (c + c) for c in cases))
    assert got == [(1, 1), (1, 7), (4, 2), (4, 5), (0, 0), (0, 0), (0, 0), (1, 1), (0, 0), (0, 0), (0, 0), (0, 0)]


def test_shared_arrays_read_as_vectors_are_declared_aligned():
    """A __shared__ array of single words that is read as float2, float4, ... has only a word's alignment of its own."""
    import re
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        text = open(os.path.join(CSRC, name)).read()
        plain = set()
        for decl in re.findall(r"^\s*__shared__\s+(?!__align__)(?:float|int|unsigned|uint32_t|uint16_t|uint8_t)\s+([^;]*);", text, re.M):
            plain |= set(re.findall(r"(\w+)\s*\[", decl))
        wide = set(re.findall(r"reinterpret_cast<(?:const )?(?:float2|float4|uint2|uint4|double|uint64_t)\s*\*>\(&?(\w+)\s*[\[+)]", text))
        assert not (plain & wide), (name, plain & wide)


def test_log_softmax_takes_clusters_for_few_long_rows_only(tmp_path):
    one = [(1, 64), (1, 8000), (64, 8000), (512, 1000), (16, 24000), (48, 48000), (256, 32000), (96, 65536)]
    eight = [(1, 12000), (12, 12000), (16, 32000), (1, 129280), (16, 160000), (64, 129280), (64, 262144)]
    got = run_cpp(tmp_path, "sample_route.h", "\n".join('printf("%%d\\n", (int)log_softmax_by_cluster(%d, %d, 148));' % c for c in one + eight))
    assert got == [(0,)] * len(one) + [(1,)] * len(eight)


def test_sampling_topk_takes_clusters_for_few_rows_that_fit_in_registers(tmp_path):
    groups = [(1, 16384), (1, 163841), (33, 64999), (64, 32000), (65, 129280)]
    clusters = [(1, 16385), (1, 163840), (32, 17000), (33, 65000), (64, 129280)]
    got = run_cpp(tmp_path, "sample_route.h", "\n".join('printf("%%d\\n", (int)topk_by_cluster(%d, %d));' % c for c in groups + clusters))
    assert got == [(0,)] * len(groups) + [(1,)] * len(clusters)


def test_sampling_topk_of_few_logits_or_several_waves_keeps_the_groups(tmp_path):
    groups = [(1, 129280, 1), (2, 100000, 1), (1, 160000, 1), (16, 16385, 1), (16, 32000, 8), (16, 100000, 1), (24, 20000, 1), (32, 32000, 8),
              (32, 100000, 1), (48, 100000, 1), (64, 100000, 8), (18, 66000, 16)]
    clusters = [(1, 16385, 1), (1, 65536, 1), (15, 65536, 2), (12, 163840, 1), (24, 65536, 8), (1, 100000, 16), (12, 129280, 8), (16, 16385, 64),
                (24, 129280, 64), (32, 22000, 64), (48, 131072, 32)]
    got = run_cpp(tmp_path, "sample_route.h", "\n".join('printf("%%d\\n", (int)topk_by_cluster(%d, %d, %d));' % c for c in groups + clusters))
    assert got == [(0,)] * len(groups) + [(1,)] * len(clusters)


def test_sampling_topk_lets_few_values_through_its_threshold(tmp_path):
    """g granules of 128 values in random order of which h reach T: about -g ln(1 - h / g) values do.  The list holds 256."""
    import math
    g = 16385 // 128 + 1
    for k, (h,) in enumerate(run_cpp(tmp_path, "sample_route.h", 'for (unsigned k = 1; k <= 64; k++) printf("%u\\n", topk_enough(k));'), 1):
        assert k <= h and -g * math.log(1 - min(h, g - 1e-9) / g) <= 200, (k, h)


def test_router_takes_a_block_per_token_while_blocks_run_at_once(tmp_path):
    warp = [(1193, 48), (1185, 47), (1300, 384), (1500, 8), (1776, 128), (2048, 16), (2049, 384), (8192, 512)]
    block = [(1, 8), (1184, 16), (1192, 512), (1800, 48), (2048, 384)]
    got = run_cpp(tmp_path, "router_route.h", "\n".join('printf("%%d\\n", (int)router_block_per_token(%d, %d));' % c for c in warp + block))
    assert got == [(0,)] * len(warp) + [(1,)] * len(block)


def test_two_tokens_keep_the_two_column_kernel_where_it_ends_sooner(tmp_path):
    Q8_0, Q5_K, Q6_K, IQ2, IQ1, IQ4 = 8, 13, 14, 16, 19, 20
    columns = [(Q8_0, 512, 12288), (Q5_K, 512, 8192), (IQ4, 512, 12288), (Q6_K, 512, 12288), (Q8_0, 16384, 1536), (Q6_K, 16384, 2048),
               (Q6_K, 8192, 8192), (IQ1, 16384, 8192), (IQ2, 8192, 4096), (Q5_K, 8192, 12288), (Q5_K, 4096, 1024)]
    mma = [(IQ1, 512, 12288), (Q8_0, 512, 4096), (Q6_K, 512, 8192), (Q6_K, 2048, 2048), (Q8_0, 32768, 4096), (Q5_K, 32768, 8192),
           (IQ4, 32768, 12288), (IQ1, 32768, 12288), (IQ2, 4096, 8192), (Q6_K, 9000, 5120), (Q8_0, 2048, 1024)]
    got = run_cpp(tmp_path, "matvec_route.h", "\n".join('printf("%%d\\n", (int)two_tokens_by_mma(%d, %d, %d, 148));' % c for c in columns + mma))
    assert got == [(0,)] * len(columns) + [(1,)] * len(mma)

