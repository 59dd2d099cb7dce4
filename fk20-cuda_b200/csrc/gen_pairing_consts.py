#!/usr/bin/env python3
"""Writes pairing_consts.inc, the precomputed constants of kernels_pairing.cu:
the Frobenius coefficients of Fp12 = Fp2[w]/(w^6 - xi), xi = 1 + u, in
Montgomery form (R = 2^384) as little-endian 32-bit limbs; and, for the
interpolation of check_proof_multi, the inverse powers of the 32nd root of
unity w32 = 5^((r - 1)/32) of Fr (the root of get_root_of_unity,
FK20Py/kzg_proofs.py:39-44) and 1/l for l = 1, 2, ..., 32, in Fr's
Montgomery form (R = 2^256).

  a^p     = sum_k conj(a_k) * g1_k w^k,  g1_k = xi^(k (p - 1) / 6)
  a^(p^2) = sum_k a_k * g2_k w^k,        g2_k = xi^(k (p^2 - 1) / 6)

It also checks the decomposition of the final exponent the kernel uses
(the hard part of the BLS12 final exponentiation, computed with exponents
z = -0xd201000000010000 and p): 3 (p^4 - p^2 + 1) / r
= (z - 1)^2 (z + p) (z^2 + p^2 - 1) + 3.
Run from this directory: python gen_pairing_consts.py > pairing_consts.inc"""
P = 0x1A0111EA397FE69A4B1BA7B6434BACD764774B84F38512BF6730D2A0F6B0F6241EABFFFEB153FFFFB9FEFFFFFFFFAAAB
R = 0x73EDA753299D7D483339D80809A1D80553BDA402FFFE5BFEFFFFFFFF00000001
Z = -0xD201000000010000
G2 = (0x024AA2B2F08F0A91260805272DC51051C6E47AD4FA403B02B4510B647AE3D1770BAC0326A805BBEFD48056C8C121BDB8,
      0x13E02B6052719F607DACD3A088274F65596BD0D09920B61AB5DA61BBDC7F5049334CF11213945D57E5AC7D055D042B7E,
      0x0CE5D527727D6E118CC9CDC6DA2E351AADFD9BAA8CBDD3A76D429A695160D12C923AC9CC3BACA289E193548608B82801,
      0x0606C4A02EA734CC32ACD2B02BC28B99CB3E287E85A763AF267492AB572E99AB3F370D275CEC1DA1AAA9075FF05F79BE)
assert (P ** 12 - 1) % R == 0 and (P ** 4 - P ** 2 + 1) % R == 0
assert 3 * (P ** 4 - P ** 2 + 1) // R == (Z - 1) ** 2 * (Z + P) * (Z ** 2 + P ** 2 - 1) + 3


def f2mul(a, b):
    return ((a[0] * b[0] - a[1] * b[1]) % P, (a[0] * b[1] + a[1] * b[0]) % P)


def f2pow(a, e):
    r = (1, 0)
    for bit in bin(e)[2:]:
        r = f2mul(r, r)
        if bit == "1":
            r = f2mul(r, a)
    return r


def limbs(x):
    m = x * 2 ** 384 % P
    return ", ".join(f"0x{(m >> (32 * i)) & 0xFFFFFFFF:08x}u" for i in range(12))


def fr_limbs(x):
    m = x * 2 ** 256 % R
    return ", ".join(f"0x{(m >> (32 * i)) & 0xFFFFFFFF:08x}u" for i in range(8))


def table(name, e):
    out = [f"__device__ const uint32_t {name}[6][2][12] = {{"]
    for k in range(6):
        g = f2pow((1, 1), k * e // 6)
        out.append(f"    {{{{{limbs(g[0])}}},\n     {{{limbs(g[1])}}}}},")
    out.append("};")
    return "\n".join(out)


print("// generated by gen_pairing_consts.py: Frobenius coefficients of Fp12, Fr roots and inverses (Montgomery form)")
print(table("c_frob1", P - 1))
print(table("c_frob2", P * P - 1))
w32 = pow(5, (R - 1) // 32, R)
assert pow(w32, 16, R) == R - 1
print("__device__ const uint32_t c_w32_inv[32][8] = {")
for k in range(32):
    print(f"    {{{fr_limbs(pow(w32, (32 - k) % 32, R))}}},")
print("};")
print("__device__ const uint32_t c_g2_gen[4][12] = {  // the G2 generator's x and y")
for v in G2:
    print(f"    {{{limbs(v)}}},")
print("};")
print("__device__ const uint32_t c_inv_pow2[6][8] = {")
for j in range(6):
    print(f"    {{{fr_limbs(pow(2 ** j, R - 2, R))}}},")
print("};")
