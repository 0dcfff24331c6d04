"""Which prompts go to pairs of CTAs, from the library's own source, against what prompts took on a B200."""

import ctypes
import subprocess
from pathlib import Path

import pytest

from megabake_b200.build import find_nvcc

SOURCE = Path(__file__).resolve().parent / "prompt_line.cu"
# us a prompt of (shape, tokens): before there were narrow pairs, now with CTAs on their own, now with narrow pairs; taken in turn
MEASURED = [
    ("1.7B", 1, 1254.4, 1225.6, 1268.8), ("1.7B", 2, 1315.8, 1272.8, 1225.2), ("1.7B", 8, 1247.2, 1209.4, 1212.4),
    ("1.7B", 16, 1271.8, 1236.0, 1239.1), ("1.7B", 24, 1269.6, 1244.2, 1217.6), ("1.7B", 32, 1260.6, 1229.9, 1224.8),
    ("1.7B", 40, 1259.5, 1241.2, 1233.4), ("1.7B", 48, 1275.9, 1250.4, 1235.5), ("1.7B", 56, 1277.1, 1252.3, 1243.1),
    ("1.7B", 64, 1274.4, 1249.3, 1241.1), ("1.7B", 65, 1457.7, 1494.0, 1383.3), ("1.7B", 72, 1517.1, 1428.0, 1385.0),
    ("1.7B", 80, 1501.5, 1412.1, 1360.9), ("1.7B", 96, 1457.2, 1420.2, 1379.2), ("1.7B", 100, 1477.7, 1434.5, 1370.7),
    ("1.7B", 112, 1501.1, 1434.6, 1387.4), ("1.7B", 128, 1473.5, 1447.0, 1391.7), ("135M", 1, 919.1, 870.4, 878.1), ("135M", 2, 906.2, 878.6, 874.4),
    ("135M", 8, 914.5, 879.6, 887.9), ("135M", 16, 943.1, 896.9, 918.1), ("135M", 24, 956.4, 918.6, 927.8), ("135M", 32, 963.1, 921.2, 933.8),
    ("135M", 40, 996.4, 950.2, 951.3), ("135M", 48, 982.0, 945.2, 950.8), ("135M", 56, 985.1, 955.4, 952.2), ("135M", 64, 995.8, 954.3, 958.4),
    ("135M", 65, 1124.3, 1081.3, 1020.5), ("135M", 72, 1127.5, 1079.2, 1015.8), ("135M", 80, 1127.4, 1081.9, 1027.1),
    ("135M", 96, 1080.2, 1040.3, 1020.9), ("135M", 100, 1104.4, 1060.9, 1027.2), ("135M", 112, 1081.4, 1034.4, 1026.1),
    ("135M", 128, 1089.5, 1037.3, 1030.0), ("0.5B", 1, 1014.4, 969.2, 977.9), ("0.5B", 2, 1027.1, 974.8, 958.5), ("0.5B", 8, 1013.7, 966.6, 959.5),
    ("0.5B", 16, 1021.9, 980.0, 976.8), ("0.5B", 24, 1028.2, 988.3, 972.8), ("0.5B", 32, 1022.4, 990.2, 977.0), ("0.5B", 40, 1090.5, 1070.1, 1002.9),
    ("0.5B", 48, 1056.8, 1023.1, 998.5), ("0.5B", 56, 1039.4, 1015.7, 987.0), ("0.5B", 64, 1043.5, 1014.8, 993.2),
    ("0.5B", 65, 1250.3, 1206.7, 1094.3), ("0.5B", 72, 1266.7, 1223.8, 1129.3), ("0.5B", 80, 1103.3, 1057.4, 1023.0),
    ("0.5B", 96, 1103.8, 1053.8, 1021.0), ("0.5B", 100, 1106.0, 1069.6, 1027.1), ("0.5B", 112, 1116.7, 1068.6, 1040.3),
    ("0.5B", 128, 1121.9, 1090.1, 1044.4), ("8B, 8 layers", 1, 983.4, 988.2, 981.5), ("8B, 8 layers", 2, 988.2, 976.2, 988.1),
    ("8B, 8 layers", 8, 982.6, 972.4, 975.9), ("8B, 8 layers", 16, 996.7, 985.6, 976.4), ("8B, 8 layers", 24, 996.4, 986.0, 976.4),
    ("8B, 8 layers", 32, 999.9, 986.7, 977.9), ("8B, 8 layers", 40, 1023.6, 1010.7, 997.4), ("8B, 8 layers", 48, 1026.0, 1016.2, 994.8),
    ("8B, 8 layers", 56, 1031.7, 1025.5, 1002.6), ("8B, 8 layers", 64, 1039.8, 1025.0, 1010.7), ("8B, 8 layers", 65, 1117.6, 1099.3, 1068.5),
    ("8B, 8 layers", 72, 1121.8, 1102.2, 1072.7), ("8B, 8 layers", 80, 1130.5, 1117.2, 1091.0), ("8B, 8 layers", 96, 1153.6, 1132.0, 1099.9),
    ("8B, 8 layers", 100, 1160.9, 1141.1, 1106.9), ("8B, 8 layers", 112, 1170.0, 1151.4, 1123.3), ("8B, 8 layers", 128, 1192.9, 1174.0, 1135.2)]


@pytest.fixture(scope="module")
def on_pairs(tmp_path_factory):
    library = tmp_path_factory.mktemp("line") / "line.so"
    subprocess.run([find_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17", "--extended-lambda", "-shared", "-Xcompiler",
                    "-fPIC", "-o", str(library), str(SOURCE)], check=True, capture_output=True, text=True)
    return ctypes.CDLL(str(library)).on_pairs


def test_no_prompt_is_slower_than_before_there_were_narrow_pairs(on_pairs):
    for shape, tokens, before, own, pairs in MEASURED:
        taken = pairs if on_pairs(0, tokens, 148) else own
        assert taken <= 1.005 * before, f"{shape}, {tokens} tokens"
    for shape, tokens, before, own, pairs in MEASURED:
        if tokens > 64:
            assert on_pairs(0, tokens, 148) and pairs < own, f"{shape}, {tokens} tokens"


def test_prompts_of_one_block_of_64_rows_are_summed_by_one_cta(on_pairs):
    """Up to 64 tokens a projection's sums keep the order they have without pairs, from 65 on q/k/v, gate/up and the head change it,
    beyond 128 tokens all do; a handle with one SM has no pairs."""
    for kind, name in enumerate(("qkv", "o", "gate and up", "down", "head")):
        for tokens in (1, 2, 16, 33, 63, 64):
            assert not on_pairs(kind, tokens, 148), name
        for tokens in (65, 100, 128):
            assert bool(on_pairs(kind, tokens, 148)) == (kind in (0, 2, 4)), name
        for tokens in (129, 256, 257, 2048):
            assert on_pairs(kind, tokens, 148), name
        for tokens in (1, 64, 65, 128, 129, 2048):
            assert not on_pairs(kind, tokens, 1), name
