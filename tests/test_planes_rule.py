"""Which calls run over whole rank planes, and which of their products on the tensor cores: a shape on either side of each line of the rules."""
import ctypes

import pytest

FORMS = ["one", "two", "grads", "conv", "step", "saved", "filter", "saved3", "filter3", "conv, plane kept", "filter from planes"]   # bits of b200cp_test_planes_choice

# what a line decides, a shape (N, C, T, H, W, R) past it and one before
LINES = [
    # up to 16 ranks: channels per pixel, and where the width is one of the row stream's (8 modulo 16) channels
    ("conv", (2, 45, 45, 10, 12, 8), (2, 45, 44, 10, 12, 8)), ("conv", (2, 45, 45, 8, 12, 16), (2, 45, 44, 8, 12, 16)),
    ("conv", (1, 144, 136, 6, 24, 12), (1, 136, 136, 6, 24, 12)), ("conv", (1, 49, 49, 9, 9, 16), (1, 49, 48, 9, 9, 16)),
    ("conv", (54, 160, 160, 24, 24, 16), (56, 160, 160, 24, 24, 16)),
    ("step", (2, 38, 38, 9, 9, 8), (2, 38, 37, 9, 9, 8)), ("step", (1, 39, 39, 8, 8, 16), (1, 39, 38, 8, 8, 16)),
    ("step", (4, 70, 70, 20, 20, 8), (3, 70, 70, 20, 20, 8)), ("step", (4, 70, 70, 20, 20, 8), (4, 68, 66, 20, 20, 8)), ("step", (1, 55, 55, 8, 8, 8), (1, 55, 54, 8, 8, 8)),
    ("step", (400, 125, 126, 7, 7, 8), (410, 125, 126, 7, 7, 8)), ("step", (410, 165, 165, 10, 14, 8), (410, 165, 165, 11, 13, 8)),
    ("step", (400, 30, 30, 7, 7, 16), (410, 30, 30, 7, 7, 16)), ("step", (20, 32, 32, 36, 34, 16), (20, 32, 32, 35, 35, 16)),
    ("step", (2, 9, 9, 9, 9, 16), (2, 9, 8, 9, 9, 16)), ("saved", (1, 36, 35, 8, 8, 16), (1, 35, 35, 8, 8, 16)),
    ("filter", (1, 11, 11, 9, 9, 8), (1, 11, 10, 9, 9, 8)), ("filter", (1, 18, 17, 9, 9, 16), (1, 17, 17, 9, 9, 16)),
    # more ranks: channels, alone or with the pixels
    ("conv", (1, 112, 112, 64, 64, 24), (1, 112, 111, 64, 64, 24)), ("conv", (1, 112, 112, 64, 64, 24), (1, 112, 112, 63, 63, 24)),
    ("conv", (1, 144, 80, 64, 64, 24), (1, 144, 80, 63, 63, 24)), ("conv", (1, 145, 79, 63, 63, 24), (1, 144, 79, 63, 63, 24)),
    ("conv", (1, 145, 79, 99, 99, 24), (1, 145, 79, 100, 100, 24)), ("conv", (1, 128, 128, 9, 9, 24), (1, 128, 127, 9, 9, 24)),
    ("conv", (32, 112, 111, 28, 28, 17), (32, 111, 111, 28, 28, 17)),
    ("conv", (1, 50, 50, 5, 5, 40), (1, 50, 49, 5, 5, 40)), ("conv", (1, 32, 70, 5, 5, 40), (1, 31, 71, 5, 5, 40)),
    ("conv", (1, 70, 32, 5, 5, 40), (1, 71, 31, 5, 5, 40)), ("conv", (1, 9, 120, 5, 5, 40), (1, 9, 119, 5, 5, 40)),
    ("conv", (10, 48, 48, 35, 36, 40), (10, 47, 47, 35, 36, 40)),
    ("step", (50, 40, 40, 21, 22, 18), (60, 40, 40, 21, 22, 18)), ("step", (60, 100, 100, 21, 22, 18), (60, 40, 40, 21, 22, 18)),
    ("step", (60, 51, 51, 21, 22, 18), (60, 51, 49, 21, 22, 18)), ("step", (60, 40, 40, 21, 24, 18), (60, 40, 40, 21, 22, 18)),
    ("filter", (1, 40, 40, 9, 9, 20), (1, 40, 39, 9, 9, 20)), ("filter", (18, 40, 39, 24, 25, 20), (18, 39, 39, 24, 25, 20)),
    ("filter", (1, 24, 24, 9, 9, 40), (1, 24, 23, 9, 9, 40)),
    # a layer: its convolution by the values in and out where the line above is of launches, older lines elsewhere
    ("conv, plane kept", (16, 170, 170, 39, 48, 16), (16, 170, 170, 38, 48, 16)), ("conv, plane kept", (32, 224, 224, 28, 28, 8), (2, 45, 45, 10, 12, 8)),
    ("conv, plane kept", (1, 49, 49, 9, 9, 16), (1, 49, 48, 9, 9, 16)), ("conv, plane kept", (1, 128, 128, 9, 9, 24), (1, 128, 127, 9, 9, 24)),
    ("conv, plane kept", (1, 65, 64, 5, 5, 40), (1, 64, 64, 5, 5, 40)), ("filter from planes", (1, 16, 16, 9, 9, 16), (1, 16, 15, 9, 9, 16)),
    ("filter from planes", (1, 65, 64, 9, 9, 20), (1, 64, 64, 9, 9, 20)),
    # products on the tensor cores: channels, pixels, the longest sum, multiply-adds
    ("one", (16, 40, 25, 8, 8, 33), (16, 40, 24, 8, 8, 33)), ("one", (13, 17, 16, 9, 9, 40), (13, 16, 16, 9, 9, 40)),
    ("one", (1, 17, 16, 8, 8, 65), (1, 16, 16, 8, 8, 65)), ("one", (13, 25, 25, 9, 9, 40), (12, 25, 25, 9, 9, 40)),
    ("one", (1, 7168, 24, 20, 20, 65), (1, 7169, 24, 20, 20, 65)), ("one", (64, 384, 384, 14, 14, 32), (64, 320, 320, 14, 14, 32)),
    ("one", (64, 512, 512, 13, 13, 18), (32, 32, 32, 39, 39, 24)),
    # two of about as many channels
    ("two", (45, 96, 144, 14, 14, 32), (44, 96, 144, 14, 14, 32)), ("two", (45, 96, 144, 14, 14, 32), (45, 96, 145, 14, 14, 32)),
    ("two", (45, 96, 144, 14, 14, 32), (45, 95, 142, 14, 14, 32)), ("two", (1, 7168, 7168, 20, 20, 32), (1, 7169, 7169, 20, 20, 32)),
    # gradients: ranks, 16-byte loads, channels
    ("grads", (1, 8, 8, 4, 4, 17), (1, 8, 8, 4, 4, 16)), ("grads", (64, 256, 256, 51, 51, 32), (64, 256, 256, 15, 15, 32)),
    ("grads", (1, 17, 16, 8, 8, 65), (1, 16, 16, 8, 8, 65)),
]


def chosen(shape):
    from paralleltnnlayers_b200._lib import TensorShape, lib
    N, C, T, H, W, R = shape
    bits = lib.b200cp_test_planes_choice(ctypes.byref(TensorShape(N=N, H=H, W=W, pad=1, T=T, C=C, Y=3, X=3, Rank=R)))
    return {name for i, name in enumerate(FORMS) if bits >> i & 1}


@pytest.mark.parametrize("what, past, before", LINES, ids=str)
def test_both_sides_of_a_line(lib_built, what, past, before):
    assert what in chosen(past) and what not in chosen(before)
