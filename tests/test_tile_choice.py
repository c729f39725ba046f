"""The choice of a tile kernel for plain bf16 products, compiled as host code, against measured times."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
WIDTHS = (192, 224, 256, 288, 320, 352, 384, 416, 448, 480, 512)
# (m, n, k) and the time of every pair width in us, medians of five runs on one B200. K is made of 64s, of 16s or of neither
MEASURED = [
    ((3448, 12576, 6360), (611.6, 586.7, 578.1, 534.1, 540.1, 507.8, 501.8, 485.3, 495.4, 499.5, 450.3)),
    ((1358, 12120, 4480), (133.7, 133.8, 113.9, 134.1, 160.7, 124.5, 145.2, 149.4, 161.1, 168.7, 129.5)),
    ((1012, 8200, 4104), (82.6, 67.5, 71.0, 73.0, 83.7, 85.6, 94.4, 89.2, 92.7, 58.6, 59.2)),
    ((8119, 560, 4720), (50.4, 54.3, 58.3, 40.3, 44.0, 47.3, 49.3, 54.5, 56.8, 57.7, 60.3)),
    ((957, 24464, 2480), (98.3, 95.6, 106.6, 113.1, 121.6, 115.5, 118.4, 125.5, 107.7, 121.1, 119.1)),
    ((1180, 13120, 5408), (135.4, 130.9, 146.6, 182.8, 152.7, 157.7, 167.7, 178.7, 194.0, 142.4, 148.4)),
    ((998, 9128, 5104), (84.0, 89.7, 68.2, 83.2, 93.1, 88.0, 99.8, 107.6, 109.8, 123.5, 76.4)),
    ((3963, 12056, 720), (75.0, 77.0, 75.5, 85.4, 88.5, 85.2, 81.9, 86.8, 88.3, 90.2, 86.0)),
    ((3039, 3016, 11624), (248.5, 261.4, 205.8, 231.8, 211.1, 223.9, 236.5, 238.4, 253.5, 267.7, 145.3)),
    ((5200, 24872, 864), (203.5, 210.1, 195.3, 248.9, 250.1, 245.7, 257.4, 247.2, 270.8, 242.1, 274.1)),
    ((7082, 896, 3936), (41.2, 48.6, 51.8, 60.1, 59.2, 65.5, 69.9, 72.8, 47.0, 47.4, 52.4)),
]

# few rows: the kernels within 15 % of the best one, us in a graph of many. 64 / 128 / 129: one-CTA tiles 64, 128 and 256 wide; 2, 192 ... 512: pair tiles; 1000 * S + BT: split-K
FEW_ROWS = [
    ((71, 3728, 11960), {8128: 24.7, 7128: 26.5, 6128: 28.4}),
    ((365, 3120, 2880), {64: 11.7, 128: 12.8}),
    ((193, 4512, 2624), {64: 11.0, 128: 12.4}),
    ((372, 2176, 4400), {5128: 16.3, 64: 16.9, 4128: 17.4, 3256: 17.5}),
    ((195, 4512, 7360), {3256: 21.9, 64: 24.2, 2064: 24.5}),
    ((329, 17224, 5424), {480: 67.3, 2: 70.4, 512: 70.9}),
    ((77, 5384, 8352), {6128: 21.0, 5128: 21.8, 4128: 23.3}),
    ((155, 22656, 2296), {320: 28.8, 352: 29.2, 384: 30.2, 416: 31.7, 448: 32.9, 192: 33.1}),
    ((65, 7448, 1472), {64: 7.7, 128: 8.7}),
    ((226, 4248, 5104), {3256: 18.6, 64: 19.0, 4128: 19.4}),
    ((438, 2136, 2280), {64: 14.0, 4128: 14.8, 3256: 15.1}),
    ((441, 2744, 10248), {3256: 39.1}),
    ((138, 12032, 3264), {192: 19.9, 224: 20.9, 1064: 22.2, 2: 22.3}),
    ((389, 976, 7744), {4064: 15.1, 6256: 15.4, 5064: 15.7, 8128: 15.7, 7128: 16.4, 5256: 16.4, 6128: 17.1}),
    ((233, 4184, 10064), {4256: 25.5}),
    ((192, 4672, 3840), {64: 14.4, 3256: 14.9, 2064: 15.4}),
    ((298, 2968, 8208), {64: 27.5, 3128: 30.0, 2064: 30.5, 5256: 31.4}),
    ((317, 3120, 9008), {64: 29.7, 3128: 32.3}),
    ((300, 2864, 3888), {64: 14.9, 4128: 16.3}),
    ((275, 3096, 2096), {64: 9.6}),
    ((282, 3128, 4704), {64: 16.9, 2064: 18.5, 3128: 19.3}),
    ((343, 3032, 5328), {64: 19.2}),
]

# the same for up to 64 rows and for more than 512: ((m, n, k, block-scaled), {1000 * S + BT: us, 0 = the tile kernels}), the kernels within 15 % of the best one
SPLITS = [
    ((25, 6400, 4400, 0), {4032: 13.1, 5032: 13.1, 3032: 13.7}),
    ((32, 14928, 592, 0), {1032: 7.0, 2032: 7.5}),
    ((2, 10688, 1320, 0), {3016: 9.2, 2016: 9.9, 1016: 10.4}),
    ((1, 13696, 1592, 0), {2016: 11.1, 1016: 12.5}),
    ((2, 26320, 8376, 0), {4016: 72.4, 5016: 73.4, 2016: 74.1, 6016: 77.0, 8016: 77.8, 3016: 78.2, 7016: 79.5, 1016: 83.1}),
    ((28, 3816, 4920, 0), {7032: 11.1, 8032: 11.1, 6032: 11.8, 5032: 11.9}),
    ((21, 7096, 568, 0), {2032: 6.1, 1032: 6.2}),
    ((31, 1344, 1160, 0), {4032: 5.1, 3032: 5.6, 2032: 5.8}),
    ((49, 1448, 1832, 0), {7064: 6.6, 4064: 6.8, 5064: 7.2, 6064: 7.4, 3064: 7.5}),
    ((2, 9696, 3720, 0), {3016: 15.9, 2016: 16.4}),
    ((24, 640, 864, 0), {3032: 4.2, 2032: 4.4}),
    ((30, 3104, 1280, 1), {2032: 5.0, 5032: 5.1, 3032: 5.2, 4032: 5.2, 1032: 5.5}),
    ((44, 14032, 1024, 1), {1064: 7.0, 2064: 7.5}),
    ((56, 10664, 5120, 1), {3064: 13.8, 2064: 14.3}),
    ((19, 3592, 1280, 1), {2032: 5.1, 3032: 5.1, 4032: 5.1, 5032: 5.1, 1032: 5.5}),
    ((28, 16888, 1664, 1), {1032: 8.2, 2032: 9.1}),
    ((41, 11000, 4224, 1), {3064: 12.1, 2064: 12.6}),
    ((1172, 576, 7776, 0), {5256: 17.5, 4256: 18.9, 5128: 19.4}),
    ((728, 1328, 7216, 0), {4256: 19.3}),
    ((1177, 520, 10240, 0), {5256: 20.1, 5128: 21.9, 4256: 21.9}),
    ((1322, 1120, 2408, 0), {0: 17.9, 2256: 19.9}),
    ((922, 1976, 12360, 0), {2256: 69.0, 4256: 70.8}),
    ((734, 1024, 14376, 0), {5256: 34.3}),
    ((912, 536, 3512, 0), {6256: 14.2, 5256: 14.2, 4256: 15.6, 6128: 16.2}),
    ((158, 6040, 2720, 0), {2192: 14.2, 0: 14.3, 2064: 15.2, 2256: 15.7}),
    ((480, 8376, 3136, 0), {0: 23.2, 1256: 26.1}),
    ((305, 2528, 14336, 0), {3192: 28.3}),
    ((180, 5376, 14912, 0), {3192: 36.5, 3256: 40.8}),
    ((133, 7432, 5568, 0), {2192: 22.4, 2256: 25.1}),
    ((150, 7024, 10368, 0), {2192: 34.6}),
    ((205, 6528, 14656, 0), {2256: 55.0, 5256: 56.5, 4256: 62.1, 2128: 62.8}),
    ((422, 3904, 14464, 0), {2256: 53.4, 2128: 59.4}),
    ((448, 3336, 13504, 0), {2256: 48.3, 2128: 55.1}),
    ((210, 6752, 10968, 0), {2256: 61.1, 4256: 62.1}),
]

# block-scaled, more than 64 rows: -128, -192, -256 one-CTA tiles, -2192, -2256 pair tiles, else split-K as above
BLOCK_SCALED = [
    ((154, 3376, 640), {1064: 5.1, -128: 5.4, -2192: 5.7, 2064: 5.7}),
    ((167, 7656, 1024), {-128: 6.9, 1064: 7.0, -2192: 7.8, -192: 7.9}),
    ((2069, 1696, 896), {-256: 8.1, -128: 8.1, -2192: 8.4, -2256: 8.6, -192: 8.7}),
    ((646, 15008, 9984), {-2192: 95.0, -2256: 96.5, -128: 106.2, -192: 108.5}),
    ((123, 1304, 640), {1064: 4.3, 2064: 4.9}),
    ((793, 17936, 9600), {-2256: 128.3, -192: 129.0, -2192: 132.5, -128: 140.4, -256: 142.5}),
    ((3331, 960, 1664), {-192: 8.4, -2192: 8.4}),
    ((72, 7624, 512), {1064: 5.4, -128: 5.6, 1128: 5.6, 1256: 5.6, -192: 6.1, -2192: 6.1, 2064: 6.2}),
    ((5210, 12968, 7040), {-2192: 356.0, -192: 369.3, -2256: 381.1, -256: 384.0}),
    ((471, 3320, 1152), {-128: 6.9, 1064: 6.9, -2192: 7.5, -192: 7.9}),
    ((933, 4048, 2816), {-2256: 13.7, -256: 14.2, 1128: 14.5, 1256: 14.5, -128: 15.3, -2192: 15.6}),
    ((223, 904, 10368), {8064: 10.1, 7064: 10.4, 6064: 10.7, 5064: 11.0, 4064: 11.1}),
    ((98, 7352, 2432), {-128: 9.8, 2064: 9.8, 1064: 10.2, 2256: 10.2, -2192: 10.5, 4128: 10.7, -192: 11.2, 3128: 11.2}),
    ((800, 12096, 896), {-192: 13.2, -128: 14.0}),
    ((2087, 8240, 768), {-192: 18.0, -128: 18.8}),
    ((767, 4808, 9472), {-2256: 31.2, -256: 34.6}),
    ((101, 21704, 3328), {-192: 17.4, 1128: 18.8, -256: 19.6}),
    ((424, 3016, 11008), {-128: 24.5, 2256: 24.6, 2128: 25.1, -2192: 26.1}),
    ((233, 5632, 7936), {3256: 17.7, 3128: 18.2, -128: 19.5}),
    ((1394, 632, 5248), {4256: 12.0, 3256: 13.0, -128: 13.7}),
    ((748, 544, 10368), {4064: 12.2, 8256: 12.6, 7256: 13.0, 8128: 13.3, 3064: 13.6, 6256: 13.7, 7128: 13.7, 5256: 13.8}),
    ((838, 1272, 6016), {2064: 13.3, 4128: 13.5, 3256: 13.8, 3128: 14.5, -128: 15.1}),
    ((261, 22368, 11904), {-256: 93.2, -192: 101.9, -128: 104.7}),
    ((252, 18048, 1536), {-128: 11.8, -2256: 11.8, -256: 12.0, 1128: 12.0, -2192: 12.3, 1256: 12.8}),
    ((279, 10192, 2688), {-256: 14.3, -128: 15.1, 1128: 15.1, -2192: 16.1}),
]

# B stored [K, N] (input gradients), drawn from the products that the choice was measured on (384 of up to 64 rows and 570 of 65 to 1100; within 8 % of the best one for 358 and 474): as SPLITS
INPUT_GRADIENTS = [
    ((59, 2360, 18168), {8064: 26.8, 7064: 28.7, 6064: 28.7}),
    ((42, 2448, 13984), {8064: 18.1, 7064: 18.1, 6064: 18.4, 5064: 20.1}),
    ((11, 320, 1544), {6016: 3.8, 5016: 3.8, 4016: 4.1}),
    ((8, 3360, 2472), {5016: 6.6, 4016: 6.6, 7016: 6.9, 8016: 6.9, 3016: 7.1, 6016: 7.2, 2016: 7.6}),
    ((36, 1376, 1656), {6064: 5.6, 5064: 5.8, 4064: 6.1}),
    ((2, 3448, 21040), {8016: 29.0, 7016: 30.0, 5016: 30.4, 6016: 32.4}),
    ((467, 6736, 7192), {0: 46.4}),
    ((134, 1344, 14424), {8192: 16.4, 7192: 17.4, 8256: 17.9, 6192: 18.3}),
    ((883, 1696, 4360), {2192: 21.8, 0: 24.8}),
    ((289, 6208, 11728), {0: 51.0, 2128: 55.1, 1192: 58.4}),
    ((546, 560, 4168), {8192: 10.8, 6192: 11.2, 7192: 11.3, 6064: 11.5, 5064: 11.9, 5192: 12.3}),
    ((222, 4592, 11208), {3256: 37.4}),
    ((546, 480, 1480), {4064: 7.3, 5064: 7.6, 3064: 7.9, 2064: 8.0}),
    ((796, 344, 576), {0: 4.6}),
    ((69, 2248, 7216), {6192: 12.3, 5192: 13.2, 6256: 13.2}),
    ((477, 432, 9536), {8192: 12.2, 7192: 12.7, 6192: 13.1, 8064: 13.4, 7064: 13.8}),
]

# (m, ffn, k, backward) of a product with SwiGLU and whether the fused kernel is the faster one: us separate / fused
FUSED_SWIGLU = [
    ((60, 512, 256, 0), True),               # 5.5 / 5.2
    ((2048, 14336, 4096, 0), True),          # 369 / 356
    ((1000, 3584, 1024, 0), True),           # 20.0 / 19.3
    ((35, 3072, 1144, 0), False),            # 9.3 / 11.7
    ((168, 2952, 8616, 0), False),           # 39.0 / 47.4
    ((650, 136, 4528, 0), False),            # 12.9 / 18.4
    ((781, 184, 16352, 0), False),           # 20.6 / 55.5
    ((2048, 14336, 4096, 1), True),          # 253 / 214
    ((777, 14336, 4096, 1), True),           # 135 / 126
    ((300, 7168, 2048, 1), False),           # 22.8 / 24.2
    ((602, 1688, 14560, 1), False),          # 46.2 / 64.3
    ((620, 128, 13320, 1), False),           # 17.7 / 53.6
]


def _choose(tmp_path, products):
    src = tmp_path / "choose.cc"
    src.write_text('#include <cstdio>\n#include "mc2/tile_choice.h"\nint main() { unsigned long long m, n, k; while (scanf("%llu %llu %llu", &m, &n, &k) == 3) { '
                   'auto c = hccl::mc2::ChoosePlain(m, n, k, 148, true); printf("%u %d %u\\n", c.splitK.split * 1000 + c.splitK.bt, (int)c.tile.pair, c.tile.bn); } }\n')
    exe = tmp_path / "choose"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{ROOT / 'csrc'}", str(src), "-o", str(exe)], check=True, timeout=120)
    out = subprocess.run([str(exe)], input="".join(f"{m} {n} {k}\n" for m, n, k in products), capture_output=True, text=True, check=True, timeout=60)
    return [tuple(int(v) for v in line.split()) for line in out.stdout.splitlines()]


def test_chosen_width_is_within_the_noise_of_the_best(tmp_path):
    """Runs of one width differed by up to 8 % where these were measured."""
    for (shape, us), (split, pair, width) in zip(MEASURED, _choose(tmp_path, [p for p, _ in MEASURED])):
        assert not split and pair and us[WIDTHS.index(width)] <= 1.08 * min(us), (shape, width, us)


def test_few_rows_take_a_kernel_near_the_best(tmp_path):
    """Where split-K pays, with as many CTAs along K as run at once, and where 64-wide tiles do."""
    for (shape, us), (split, pair, width) in zip(FEW_ROWS, _choose(tmp_path, [p for p, _ in FEW_ROWS])):
        kernel = split or ((2 if width == 256 else width) if pair else {64: 64, 128: 128, 256: 129}[width])
        assert us.get(kernel, 1e9) <= 1.08 * min(us.values()), (shape, kernel, us)


def test_number_of_ctas_along_k(tmp_path):
    """Up to 64 rows: as many CTAs along K as the waves of clusters make good, block-scaled too. More than 512: 256-row tiles where they pay. Every choice can be launched."""
    src = tmp_path / "split.cc"
    src.write_text('#include <cstdio>\n#include "mc2/tile_choice.h"\nusing namespace hccl::mc2;\nint main() { unsigned long long m, n, k; int mx; '
                   'while (scanf("%llu %llu %llu %d", &m, &n, &k, &mx) == 4) { auto c = mx ? ChooseSplitK(m, n, k, true, false) : ChoosePlain(m, n, k, 148, true).splitK; '
                   'printf("%u\\n", c.split ? c.split * 1000 + c.bt : 0); } }\n')
    exe = tmp_path / "split"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{ROOT / 'csrc'}", str(src), "-o", str(exe)], check=True, timeout=120)

    def choose(products):
        out = subprocess.run([str(exe)], input="".join("%d %d %d %d\n" % p for p in products), capture_output=True, text=True, check=True, timeout=60)
        return [int(v) for v in out.stdout.split()]

    for (shape, us), kernel in zip(SPLITS, choose([p for p, _ in SPLITS])):
        assert us.get(kernel, 1e9) <= 1.08 * min(us.values()), (shape, kernel, us)
    every = [(m, n, k, mx) for m in (1, 16, 17, 32, 33, 64, 65, 512, 513, 4096, 100000) for n in (8, 120, 128, 4096, 128256) for k in (8, 128, 504, 512, 768, 2048, 3304, 16384)
             for mx in (0, 1) if not mx or k % 128 == 0]
    for (m, n, k, mx), kernel in zip(every, choose(every)):
        s, bt = divmod(kernel, 1000)
        assert not kernel or (1 <= s <= 8 and s * 256 <= max(k, 256) and bt in (16, 32, 64, 128, 192, 256) and (not mx or bt <= 64 and (bt == 64 or m <= bt))), (m, n, k, mx, kernel)


def test_block_scaled_products_of_many_rows(tmp_path):
    """A kernel near the best, and one that can be launched: pairs only where they are enabled and N has a tile of them, 64-row tiles from whole scale atoms on."""
    src = tmp_path / "mx.cc"
    src.write_text('#include <cstdio>\n#include "mc2/tile_choice.h"\nint main() { unsigned long long m, n, k; int pairs; while (scanf("%llu %llu %llu %d", &m, &n, &k, &pairs) == 4) { '
                   'auto c = hccl::mc2::ChooseMx(m, n, k, 148, pairs); printf("%d\\n", c.splitK.split ? (int)(c.splitK.split * 1000 + c.splitK.bt) '
                   ': c.tile.pair ? -(int)(2000 + c.tile.bn) : -(int)c.tile.bn); } }\n')
    exe = tmp_path / "mx"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{ROOT / 'csrc'}", str(src), "-o", str(exe)], check=True, timeout=120)

    def choose(products):
        out = subprocess.run([str(exe)], input="".join("%d %d %d %d\n" % p for p in products), capture_output=True, text=True, check=True, timeout=60)
        return [int(v) for v in out.stdout.split()]

    for (shape, us), kernel in zip(BLOCK_SCALED, choose([p + (1,) for p, _ in BLOCK_SCALED])):
        assert us.get(kernel, 1e9) <= 1.08 * min(us.values()), (shape, kernel, us)
    every = [(m, n, k, pairs) for m in (1, 17, 33, 64, 65, 129, 513, 4096, 100000) for n in (8, 248, 256, 4096, 128256) for k in (128, 256, 768, 2048, 16384) for pairs in (0, 1)]
    for (m, n, k, pairs), kernel in zip(every, choose(every)):
        if kernel > 0:
            s, bt = divmod(kernel, 1000)
            assert 1 <= s <= 8 and s * 128 <= k and bt in (16, 32, 64, 256) and (m <= bt or bt >= 64)
        else:
            assert kernel in (-128, -192, -256) or (kernel in (-2192, -2256) and pairs and n >= 256), (m, n, k, pairs, kernel)


def test_input_gradients_take_a_kernel_near_the_best(tmp_path):
    """B stored [K, N]: split-K where it pays, and a choice that can be launched. Where the SwiGLU layer's products are fused with it: never where the product by itself splits K, which the
    fused kernel cannot."""
    src = tmp_path / "nn.cc"
    src.write_text('#include <cstdio>\n#include "mc2/tile_choice.h"\nusing namespace hccl::mc2;\nint main() { unsigned long long m, n, k; while (scanf("%llu %llu %llu", &m, &n, &k) == 3) { '
                   'auto c = ChooseNn(m, n, k, 148, true), f = ChoosePlain(m, 2 * n, k, 148, true); printf("%u %d %u %u %u %u %u\\n", c.splitK.split * 1000 + c.splitK.bt, (int)c.tile.pair, c.tile.bn, '
                   'f.splitK.split, ChooseSwiGlu(m, n, k, false, 148, true), ChooseSwiGlu(m, n, k, true, 148, true), ChooseSwiGlu(m, n, k, true, 148, false) + ChooseSwiGlu(m, n, k, false, 148, false)); } }\n')
    exe = tmp_path / "nn"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{ROOT / 'csrc'}", str(src), "-o", str(exe)], check=True, timeout=120)

    def choose(products):
        out = subprocess.run([str(exe)], input="".join("%d %d %d\n" % p for p in products), capture_output=True, text=True, check=True, timeout=60)
        return [tuple(int(v) for v in line.split()) for line in out.stdout.splitlines()]

    for (shape, us), (kernel, *_) in zip(INPUT_GRADIENTS, choose([p for p, _ in INPUT_GRADIENTS])):
        assert us.get(kernel if kernel >= 1000 else 0, 1e9) <= 1.08 * min(us.values()), (shape, kernel, us)
    for ((m, n, k, backward), fused), c in zip(FUSED_SWIGLU, choose([p[:3] for p, _ in FUSED_SWIGLU])):
        assert bool(c[5 if backward else 4]) == fused, (m, n, k, backward, c)
    every = [(m, n, k) for m in (1, 16, 17, 40, 64, 65, 200, 512, 513, 700, 1100, 4096, 100000) for n in (8, 64, 120, 512, 3584, 14336) for k in (8, 256, 504, 512, 1024, 2048, 4096, 16384)]
    for (m, n, k), (kernel, pair, bn, splits, forward, backward, off) in zip(every, choose(every)):
        s, bt = divmod(kernel, 1000)
        assert not s or (s <= 8 and s * 256 <= k and bt in (16, 32, 64, 128, 192, 256)), (m, n, k, kernel)
        assert (pair and bn in (256, 512)) or (not pair and bn in (64, 128)), (m, n, k, pair, bn)
        assert forward in (0, 128, 192, 224, 256) and backward in (0, 128, 256) and not off
        assert not (forward and splits) and not (backward and s) and bool(forward) == (not splits) and bool(backward) == (m > 512 and not s), (m, n, k)
