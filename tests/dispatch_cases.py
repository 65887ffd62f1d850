"""Shapes by the kernel form that the library chooses for them: tests/test_host_dispatch.py asserts the choice without a GPU, the GPU
tests run the same shapes."""

# One layer (convolution of filter k, stride 1, padding k // 2, then ReLU and a pooling, so that its result stays NHWC) whose reduction
# is split: precision, (images, channels, h, w, output channels, k), CTAs of a cluster, channels of a tile. Every size of a cluster at
# every width it is chosen for; tiles of 128, 126, 121, 117, 98, 63, 9 and 1 pixels, whose rows divide unevenly among 3, 5, 6 and 7 owners
# (and among 8 when there are fewer than 8); last tiles of 32 to 96 channels.
SPLIT_LAYERS = [
    ("bf16", (50, 1024, 14, 9, 32, 1), 2, 64), ("bf16", (64, 768, 7, 7, 160, 1), 2, 128), ("bf16", (40, 768, 14, 9, 32, 1), 3, 64),
    ("bf16", (5, 768, 7, 7, 1600, 1), 3, 128), ("bf16", (28, 192, 13, 11, 160, 3), 3, 256), ("bf16", (24, 768, 14, 9, 32, 1), 4, 64),
    ("bf16", (3, 1536, 7, 7, 1600, 1), 4, 128), ("bf16", (20, 256, 13, 11, 160, 3), 4, 256), ("bf16", (24, 128, 8, 16, 32, 3), 5, 64),
    ("bf16", (5, 128, 7, 7, 1024, 3), 5, 128), ("bf16", (2, 768, 7, 7, 32, 1), 6, 64), ("bf16", (18, 128, 13, 11, 96, 3), 6, 128),
    ("bf16", (1, 192, 9, 7, 64, 3), 7, 64), ("bf16", (4, 192, 4, 6, 32, 3), 7, 64), ("bf16", (1, 192, 3, 3, 32, 3), 7, 64),
    ("bf16", (2, 1024, 7, 7, 32, 1), 8, 64), ("bf16", (1, 1024, 1, 1, 32, 1), 8, 64), ("bf16", (1, 320, 3, 3, 1600, 3), 8, 128),
    ("tf32", (50, 512, 14, 9, 32, 1), 2, 64), ("tf32", (64, 512, 7, 7, 160, 1), 2, 128), ("tf32", (64, 512, 7, 7, 320, 1), 2, 256),
    ("tf32", (40, 512, 14, 9, 32, 1), 3, 64), ("tf32", (5, 512, 7, 7, 1600, 1), 3, 128), ("tf32", (40, 512, 14, 9, 160, 1), 3, 256),
    ("tf32", (1, 512, 1, 1, 1600, 1), 4, 64), ("tf32", (3, 768, 7, 7, 1600, 1), 4, 128), ("tf32", (20, 128, 13, 11, 160, 3), 4, 256),
    ("tf32", (24, 768, 14, 9, 32, 1), 5, 64), ("tf32", (5, 768, 7, 7, 1024, 1), 5, 128), ("tf32", (40, 512, 7, 7, 32, 1), 6, 64),
    ("tf32", (11, 512, 14, 9, 224, 1), 6, 128), ("tf32", (2, 512, 7, 7, 32, 1), 8, 64), ("tf32", (28, 1536, 7, 7, 96, 1), 8, 128),
    ("tf32x3", (50, 512, 14, 9, 32, 1), 2, 64), ("tf32x3", (64, 768, 7, 7, 160, 1), 2, 128), ("tf32x3", (40, 512, 14, 9, 32, 1), 3, 64),
    ("tf32x3", (5, 512, 7, 7, 1600, 1), 3, 128), ("tf32x3", (3, 512, 7, 7, 1600, 1), 4, 128), ("tf32x3", (24, 768, 14, 9, 32, 1), 5, 64),
    ("tf32x3", (5, 768, 7, 7, 1024, 1), 5, 128), ("tf32x3", (40, 768, 7, 7, 96, 1), 6, 128), ("tf32x3", (1, 512, 1, 1, 32, 1), 8, 64),
    ("tf32x3", (28, 1024, 7, 7, 96, 1), 8, 128),
    ("bf16", (33, 512, 9, 7, 288, 3), 3, 256),
]


def split_layer(relay, case, to_constant, weight, bias):
    n, c, h, w, _, k = case
    x = relay.Var("input", (n, c, h, w))
    conv = relay.Call("nn_conv2d", [x, relay.Constant(to_constant(weight)), relay.Constant(to_constant(bias))],
                      relay.Conv2DAttrs((1, 1), (k // 2,) * 4, (1, 1), 1))
    pool = relay.MaxPool2DAttrs((1, 1), (1, 1, 1, 1), (1, 1), (3, 3), "NCHW", False)
    return relay.Function([x], relay.Call("nn_max_pool2d", [relay.Call("nn_relu", [conv])], pool))

# Convolutions of the bit-exact fp32 mode by the tile of its packed kernel: (images, channels, h, w, output channels, kh, kw, stride, pad,
# dilation), width of the filter (0: any but 1, 3 and 7), channels x pixels of a block. Every tile of every width, reductions of one stage
# up to one more than a ring holds.
FP32_TILES = [
    ((1, 3, 5, 6, 16, 3, 2, 1, 1, 1), 0, "16x32"), ((3, 3, 40, 41, 17, 3, 2, 1, 1, 1), 0, "32x64"), ((3, 3, 57, 58, 33, 3, 2, 1, 1, 1), 0, "64x96"),
    ((5, 3, 57, 58, 33, 3, 2, 1, 1, 1), 0, "64x128"), ((1, 3, 5, 6, 16, 1, 1, 1, 0, 1), 1, "16x32"), ((3, 3, 40, 41, 17, 1, 1, 1, 0, 1), 1, "32x64"),
    ((3, 40, 40, 41, 17, 1, 1, 1, 0, 1), 1, "32x64"), ((3, 3, 57, 58, 33, 1, 1, 1, 0, 1), 1, "64x96"), ((5, 3, 57, 58, 33, 1, 1, 1, 0, 1), 1, "64x128"),
    ((1, 3, 5, 6, 16, 3, 3, 1, 1, 1), 3, "16x16"), ((1, 11, 5, 6, 16, 3, 3, 1, 1, 1), 3, "16x16"), ((1, 16, 5, 6, 16, 3, 3, 1, 1, 1), 3, "16x16"),
    ((1, 21, 5, 6, 16, 3, 3, 1, 1, 1), 3, "16x16"), ((1, 32, 5, 6, 16, 3, 3, 1, 1, 1), 3, "16x16"), ((3, 3, 20, 21, 17, 3, 3, 1, 1, 1), 3, "16x32"),
    ((3, 3, 28, 29, 17, 3, 3, 1, 1, 1), 3, "32x32"), ((3, 3, 40, 41, 17, 3, 3, 1, 1, 1), 3, "32x64"), ((3, 3, 40, 41, 33, 3, 3, 1, 1, 1), 3, "32x96"),
    ((5, 3, 40, 41, 33, 3, 3, 1, 1, 1), 3, "32x128"), ((3, 3, 57, 58, 33, 3, 3, 1, 1, 1), 3, "64x96"), ((5, 3, 57, 58, 33, 3, 3, 1, 1, 1), 3, "64x128"),
    ((1, 3, 5, 6, 16, 7, 7, 1, 3, 1), 7, "16x16"), ((3, 3, 20, 21, 17, 7, 7, 1, 3, 1), 7, "16x32"), ((3, 3, 28, 29, 17, 7, 7, 1, 3, 1), 7, "32x32"),
    ((3, 3, 40, 41, 17, 7, 7, 1, 3, 1), 7, "32x64"), ((3, 3, 40, 41, 33, 7, 7, 1, 3, 1), 7, "32x96"), ((5, 3, 40, 41, 33, 7, 7, 1, 3, 1), 7, "32x128"),
    ((3, 3, 57, 58, 33, 7, 7, 1, 3, 1), 7, "64x96"),
]

# int8 filters of 81 taps, which it does not take: (images, channels, h, w, output channels, k), whether the result leaves by way of NHWC.
# Results below and from 1 MiB on, planes that are multiples of 16, of 4 and odd, channels that are multiples of 16, of 4 and odd, boxes of two
# and fewer columns and wider ones, one pixel per image.
S8_LARGE_FILTERS = [
    ((64, 20, 7, 7, 100, 9), False), ((16, 24, 14, 14, 50, 9), False), ((2, 48, 12, 12, 40, 9), False), ((5, 3, 41, 43, 33, 9), False),
    ((66, 24, 13, 13, 401, 9), True), ((256, 16, 7, 7, 30, 9), True), ((128, 17, 5, 5, 33, 9), True), ((64, 40, 7, 7, 96, 9), True),
    ((29, 12, 28, 28, 178, 9), True), ((9, 33, 30, 30, 400, 9), True), ((40, 8, 14, 14, 141, 9), True), ((4, 130, 48, 48, 128, 9), True),
]

# Convolutions that the channel-major kernel takes: precision, (images, channels, h, w, output channels, kh, kw, stride, pad, dilation),
# whether four columns leave at a time. Taps that share a box and taps that do not, two and four boxes of a stride-2 filter, groups of one
# to four taps, last channel blocks of one to four instructions, one to four chunks of columns per epilogue warp, several images per
# tile, planes of one row and of one column, one channel tile and one more channel than that.
CHMAJOR = [
    ("tf32", (9, 72, 45, 51, 120, 3, 3, 1, 1, 1), False), ("tf32", (1, 31, 3, 6, 64, 3, 3, 1, 0, 1), True), ("tf32", (9, 123, 45, 44, 93, 1, 1, 1, 0, 1), True),
    ("tf32", (16, 2, 20, 19, 257, 1, 1, 1, 0, 2), False), ("tf32", (7, 21, 51, 49, 200, 1, 1, 2, 0, 1), False), ("tf32", (16, 17, 8, 4, 128, 3, 3, 2, 2, 2), False),
    ("tf32", (3, 30, 12, 8, 100, 3, 3, 2, 1, 1), True), ("tf32", (33, 48, 22, 27, 1, 5, 5, 1, 2, 1), False), ("tf32", (2, 116, 8, 8, 129, 1, 3, 1, 0, 2), True),
    ("tf32", (3, 35, 3, 3, 64, 3, 1, 2, 2, 1), True), ("tf32", (1, 19, 17, 18, 64, 3, 3, 1, 1, 2), True), ("tf32", (1, 57, 11, 13, 128, 7, 1, 1, 2, 2), False),
    ("s8", (1, 1, 1, 1, 1, 1, 1, 1, 0, 1), False), ("s8", (300, 5, 1, 1, 40, 1, 1, 1, 0, 1), False), ("s8", (3, 128, 28, 28, 128, 3, 3, 1, 1, 1), True),
    ("s8", (2, 33, 1, 300, 7, 1, 3, 1, 1, 1), True), ("s8", (2, 70, 270, 1, 131, 3, 1, 1, 1, 1), False), ("s8", (16, 130, 7, 7, 100, 3, 3, 1, 1, 1), False),
    ("s8", (2, 40, 23, 21, 129, 3, 3, 2, 1, 1), False), ("s8", (3, 257, 30, 24, 33, 3, 3, 2, 1, 1), True), ("s8", (2, 96, 15, 17, 260, 5, 5, 1, 2, 1), False),
    ("s8", (7, 16, 9, 9, 8, 7, 7, 2, 2, 1), True), ("s8", (2, 206, 11, 12, 1, 7, 7, 1, 2, 2), True), ("s8", (2, 65, 21, 19, 64, 1, 1, 2, 0, 1), False),
    ("s8", (5, 31, 64, 64, 64, 3, 3, 1, 1, 1), True), ("s8", (1, 12, 41, 41, 129, 7, 3, 2, 3, 2), False),
]

# ... and with taps further than 2^15 pixels from their result: precision, images, channels, h, w, output channels, filter, stride, padding, dilation
CHMAJOR_FAR = [
    ("s8", 1, 16, 1, 50000, 32, (1, 3), 1, (0, 0), (1, 17000)), ("s8", 1, 16, 1, 64, 8, (1, 3), 1, (0, 33000), (1, 1)), ("s8", 1, 3, 40005, 1, 5, (3, 1), 1, (0, 0), (20000, 1)),
    ("s8", 1, 20, 3, 70003, 33, (1, 3), 2, (0, 0), (1, 34000)), ("tf32", 1, 64, 1, 50000, 128, (1, 3), 1, (0, 0), (1, 17000)),
    ("tf32", 1, 64, 1, 40000, 128, (1, 3), 1, (0, 33000), (1, 1)),
]

# Layers of a plan that it takes, NHWC results: (images, channels, h, w, output channels, k, stride). chmajor_layers is that layer, a second one
# of its output channels with the first one's result as residual (1x1, stride 1), and a pooling that keeps its result NHWC.
CHMAJOR_LAYERS = [
    ("bf16", (16, 64, 37, 35, 32, 1, 1)), ("bf16", (5, 64, 29, 26, 128, 1, 1)), ("bf16", (16, 64, 14, 10, 192, 1, 1)), ("bf16", (16, 64, 12, 19, 192, 1, 1)),
    ("bf16", (1, 64, 3, 3, 32, 3, 1)), ("bf16", (16, 128, 17, 13, 128, 1, 1)), ("bf16", (3, 64, 26, 23, 192, 3, 1)), ("bf16", (1, 64, 5, 6, 32, 3, 1)),
    ("tf32", (5, 32, 29, 26, 96, 1, 1)), ("tf32", (33, 64, 7, 9, 192, 1, 1)), ("tf32", (33, 32, 15, 14, 192, 1, 2)), ("tf32", (1, 32, 3, 3, 64, 3, 1)),
    ("tf32", (2, 32, 4, 3, 320, 3, 1)), ("tf32", (16, 32, 15, 17, 96, 3, 1)), ("tf32", (16, 32, 3, 5, 32, 3, 2)), ("tf32", (8, 32, 33, 35, 32, 5, 1)),
]


# 3x3 layers of a plan that its CTA pairs take: (images, h, w, channels, residual). pair_layers is a 1x1 layer to those channels, the 3x3 layer, with the
# first one's result as residual or without, and a pooling that keeps the result NHWC. Boxes of part of a plane and of whole ones, which share their
# padding, one and two images to a box, an odd number of boxes, and channels that leave the second CTA a part, or nothing, of a tile.
CHMAJOR_PAIRS = [("tf32", (48, 9, 9, 160, False)), ("tf32", (21, 14, 14, 160, True)), ("tf32", (47, 9, 10, 160, True)), ("tf32", (61, 7, 7, 288, True)),
                 ("bf16", (10, 14, 15, 320, True)), ("bf16", (195, 4, 4, 320, False))]
# ... of other paddings and dilations (the last two entries): no padding, in one direction or both, more than the filter's reach, taps two apart; planes in part and
# whole, two and three images to a box
CHMAJOR_PAIR_PADDINGS = [
    ("tf32", (41, 12, 15, 160, False, (0, 0), (1, 1))), ("tf32", (97, 4, 8, 160, False, (2, 2), (1, 1))), ("tf32", (13, 17, 13, 160, False, (3, 1), (1, 1))),
    ("tf32", (97, 6, 6, 160, False, (3, 1), (1, 1))), ("tf32", (97, 4, 15, 160, False, (2, 2), (2, 2))), ("tf32", (41, 12, 15, 160, False, (1, 1), (2, 2))),
    ("tf32", (25, 13, 16, 160, False, (2, 1), (2, 1))), ("tf32", (211, 2, 5, 160, False, (2, 2), (1, 1))), ("bf16", (151, 6, 5, 320, False, (0, 1), (1, 1))),
    ("bf16", (151, 4, 7, 320, False, (1, 0), (1, 1))), ("bf16", (211, 4, 4, 320, False, (2, 2), (2, 2))), ("bf16", (211, 6, 6, 320, False, (0, 0), (1, 1)))]


# Three-pass layers that pairs of the implicit-GEMM kernel take: of a plan (pair_layers), and operators (images, channels, h, w, outputs, kernel, stride, residual). An
# odd number of pixel tiles, channels that fill no tile of 64 or leave nothing to the second CTA's half of it, several tiles to a CTA and fewer than CTAs.
THREE_PASS_PAIRS = [(9, 39, 36, 64, True), (15, 40, 23, 64, False), (12, 15, 31, 160, True), (14, 25, 23, 96, True)]
THREE_PASS_OPERATORS = [(2, 81, 42, 42, 70, 3, 1, True), (7, 40, 45, 40, 33, 5, 1, False), (28, 74, 18, 19, 186, 3, 2, True), (32, 44, 11, 10, 131, 5, 1, False)]


def pair_layers(relay, case, to_constant, weights, biases):
    n, h, w, _, residual = case[:5]
    padding, dilation = case[5:] or ((1, 1), (1, 1))
    x = relay.Var("input", (n, weights[0].shape[1], h, w))
    conv = lambda d, i, p, dil: relay.Call("nn_conv2d", [d, relay.Constant(to_constant(weights[i])), relay.Constant(to_constant(biases[i]))],
                                           relay.Conv2DAttrs((1, 1), p * 2, dil, 1))
    y = relay.Call("nn_relu", [conv(x, 0, (0, 0), (1, 1))])
    z = conv(y, 1, padding, dilation)
    z = relay.Call("nn_relu", [relay.Call("add", [z, y]) if residual else z])
    return relay.Function([x], relay.Call("nn_max_pool2d", [z], relay.MaxPool2DAttrs((1, 1), (1, 1, 1, 1), (1, 1), (3, 3), "NCHW", False)))


def chmajor_layers(relay, case, to_constant, weights, biases):
    n, c, h, w, _, k, s = case
    x = relay.Var("input", (n, c, h, w))
    conv = lambda d, i, k, s: relay.Call("nn_conv2d", [d, relay.Constant(to_constant(weights[i])), relay.Constant(to_constant(biases[i]))],
                                         relay.Conv2DAttrs((s, s), (k // 2,) * 4, (1, 1), 1))
    y = relay.Call("nn_relu", [conv(x, 0, k, s)])
    z = relay.Call("nn_relu", [relay.Call("add", [conv(y, 1, 1, 1), y])])
    return relay.Function([x], relay.Call("nn_max_pool2d", [z], relay.MaxPool2DAttrs((1, 1), (1, 1, 1, 1), (1, 1), (3, 3), "NCHW", False)))
