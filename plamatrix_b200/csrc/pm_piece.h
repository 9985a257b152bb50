// Sizes of the 16-byte pieces in which arrays are copied to shared memory.
#pragma once

namespace pm
{

// Bytes to read for a piece that starts `left` > 0 elements of `size` bytes before the end of its array.
// The count is clamped before the product: from 2^28 elements of eight bytes left * size is past an int.
constexpr int piece_bytes(int left, int size)
{
    const int whole = 16 / size;
    return (left < whole ? left : whole) * size;
}

} // namespace pm
