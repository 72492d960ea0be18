"""Which form the recurrences' steps take, from host numbers alone: on each side of the lines, with what both forms were measured to take."""
import pytest

from tinyinfer_b200 import ops

ONE = [1]


@pytest.mark.parametrize("lens,heads,dim,chunked", [
    ([128], 16, 128, True),                   # us in stretches and in chunks: 86, 64
    ([127], 16, 128, False),
    (ONE * 8 + [128], 16, 128, True),         # 152, 92
    (ONE * 27 + [128], 16, 128, False),       # 162, 197
    (ONE * 27 + [512], 16, 128, True),        # 547, 199
    (ONE * 64 + [128], 16, 128, False),       # 182, 412
    (ONE * 128 + [128], 16, 128, False),      # 221, 784
    (ONE * 128 + [512], 16, 128, False),      # 610, 795
    (ONE * 128 + [512], 4, 64, True),         # 392, 111
    ([8] * 32 + [128], 32, 64, False),        # 131, 201
    ([128] * 16, 16, 128, True),              # 371, 195
    ([128] * 16, 32, 64, False),              # 158, 223
    ([512] * 8, 32, 64, True),
    (ONE * 250 + [256], 32, 64, False),       # 285, 1,278
    ([4096] * 2, 64, 128, False),             # the chunks' states would take more than their share of memory
])
def test_linear_attention_in_chunks(lens, heads, dim, chunked):
    tokens, n = sum(lens), len(lens)
    assert ops.linear_chunks(tokens, n, max(lens), heads, dim, dim) == (tokens // 64 + n if chunked else 0)


@pytest.mark.parametrize("lens,heads,dim,quads", [
    ([68], 16, 128, True),
    ([67], 16, 128, False),
    ([1000], 16, 128, True),                  # us token by token and by quads: 289, 213
    ([1000, 200, 200, 200], 16, 128, True),   # 391, 301
    ([512] * 2, 16, 128, False),              # 205, 219
    ([256] * 3, 16, 128, False),              # 141, 172
    ([16] * 64, 16, 128, False),              # 238, 270
    ([5] * 80, 16, 128, False),               # 176, 217
    ([64] * 4, 16, 128, False),               # 65, 70
    (ONE * 128 + [600], 16, 128, True),       # 424, 383
    ([1000], 32, 128, False),                 # 391, 408
    ([512] * 2, 32, 64, True),                # 164, 119
    ([512] * 8, 32, 64, False),               # 389, 434
    ([512] * 8, 4, 64, True),                 # 143, 102
    ([128], 8, 256, False),                   # 70, 76
    ([1000], 8, 256, True),                   # 431, 395
    ([512] * 2, 8, 256, True),                # 500, 406
    ([256] * 3, 8, 256, False),               # 299, 314
])
def test_delta_rule_by_quads(lens, heads, dim, quads):
    assert ops.delta_quads_pay(lens, heads, dim, dim) is quads


@pytest.mark.parametrize("decoded,keys,portion,apart", [
    (1, 1024, [512], False),                  # us together and apart: 66, 68
    (1, 2048, [512], True),                   # 117, 72
    (1, 8192, [64], True),                    # 86, 61
    (1, 2048, [64], False),                   # 43, 49
    (8, 4096, [8], False),                    # 55, 66
    (16, 2048, [8], True),                    # 62, 57
    (27, 4096, [60, 4], True),                # 221, 107
    (27, 4096, [], False),                    # decoded tokens alone
    (0, 0, [64, 300], False),
])
def test_decoded_tokens_beside_a_portion_of_latent_attention(decoded, keys, portion, apart):
    lens = [1] * decoded + portion
    starts = [keys - 1] * decoded + [0] * len(portion)
    assert ops.latent_decoded_apart(lens, starts) == (decoded if apart else 0)
    assert ops.latent_decoded_apart(portion + [1] * decoded, [0] * len(portion) + [keys - 1] * decoded) == 0     # not ahead of the portions
