// bsa_atable64_tc.cu -- the FP64 A(f) table on the tensor cores.
//
// A(f)[(itc, i)][m] = s_i sum_j c_ij^|f| s_j L[(itc, j)][m], s = sqrt(S(f)), as k_atable
// (bsa_kernels.cu), whose FP64 pipe (two lanes an SM and clock) spends 10 instructions on each
// c_ij^|f| and one per mode on its products.  Here the coherence is formed in integers and the sum is
// an error-free digit product (bsa_pair64_tc.cu):
//   * t = -|f| log2 c in 57 fraction bits (one FP64 multiply and one conversion), 2^-t = 2^-n T1[k1]
//     T2[k2] (1 - e): two tables of 2^(-k / 256) and 2^(-k / 65536) in 63 bits and
//     e = x - x^2/2 + x^3/6, x < 2^-16 ln 2, in 64-bit integer products; the next term is below 2^-70;
//   * c_ij^|f| <= 1 and c_ii = 1, so the row scale is 1: eight balanced base-256 digits of its 62
//     fraction bits go straight to shared memory as bf16;
//   * B = s_j L_jm has its digits prepared per frequency and component (k_wexp, k_wdigits), its column
//     scale from the exponents.
// One block per (f, itc, 128 rows): 16 warps generate digits of 32 columns at a time into two halves of
// the A tiles and drain TMEM at the end, one thread loads B and issues the MMAs.  Bound by the integer
// instructions of the generation (about 110 an element).  65 rows of 400 nodes x 2, 24 modes: FP64 pipe
// 1.70 ms, here 0.25, 0.04 for the B digits and 0.04 for the elements far below their column's scale,
// which k_atable64_mend sums on the FP64 pipe; 3333 rows of 150 nodes, 12 modes: 3.9 ms, here 1.13, 0.09 and
// 0.08.  Coherences outside [0, 1] or c_ii != 1 (bad flag of the coherence table) leave the table to k_atable.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "bsa_digits.cuh"
#include "bsa_kernels.cuh"
#include "bsa_pair64.cuh"
#include "bsa_tc.cuh"

namespace bsa {
namespace at64 {

using namespace tc;
using namespace p64;

// round(2^(63 - k / 256)) and round(2^(63 - k / 65536)), k = 0 .. 255
__device__ const unsigned long long kPow2[2][256] = {
    {0x8000000000000000ull, 0x7fa765aca88f6453ull, 0x7f4f08ae3dc7c426ull, 0x7ef6e8da4b544f9aull,
     0x7e9f06067a4360baull, 0x7e47600890f223deull, 0x7deff6b672f84e24ull, 0x7d98c9e62113e1faull,
     0x7d41d96db915019dull, 0x7ceb252375c9cf9bull, 0x7c94acddaeea5d3aull, 0x7c3e7072d904a6ceull,
     0x7be86fb985689ddcull, 0x7b92aa886214411cull, 0x7b3d20b6399fc237ull, 0x7ae7d219f329b948ull,
     0x7a92be8a92436616ull, 0x7a3de5df36dcfeefull, 0x79e947ef1d320d2dull, 0x7994e4919db5d74eull,
     0x7940bb9e2cffd89dull, 0x78ecccec5bb84661ull, 0x78991853d684a285ull, 0x78459dac65f45bb5ull,
     0x77f25ccdee6d7ae6ull, 0x779f559070195e36ull, 0x774c87cc06d1812eull, 0x76f9f358ea0c5249ull,
     0x76a7980f6cca15c2ull, 0x765575c7fd81d5a0ull, 0x76038c5b260e5eeeull, 0x75b1dba18b9b4c20ull,
     0x75606373ee921c97ull, 0x750f23ab2a87593eull, 0x74be1c203627c62bull, 0x746d4cac2325a155ull,
     0x741cb5281e25ee34ull, 0x73cc556d6eadce5full, 0x737c2d55770fe711ull, 0x732c3cb9b459d38bull,
     0x72dc8373be41a454ull, 0x728d015d47136b40ull, 0x723db6501b9ed447ull, 0x71eea2262324cb0cull,
     0x719fc4b95f452d29ull, 0x71511de3ebec8913ull, 0x7102ad7fff41e9b4ull, 0x70b47367e994ae92ull,
     0x70666f76154a7089ull, 0x7018a18506ccf314ull, 0x6fcb096f5c782210ull, 0x6f7da70fce881bf9ull,
     0x6f307a412f074892ull, 0x6ee382de69bc7bf8ull, 0x6e96c0c284192610ull, 0x6e4a33c89d278e49ull,
     0x6dfddbcbed791babull, 0x6db1b8a7c714a92bull, 0x6d65ca379564e639ull, 0x6d1a1056dd26c382ull,
     0x6cce8ae13c57ebdbull, 0x6c8339b26a25494eull, 0x6c381ca636d99642ull, 0x6bed33988bcbfab5ull,
     0x6ba27e656b4eb57aull, 0x6b57fce8f09dd17full, 0x6b0daeff4fcde703ull, 0x6ac39484d5bae8c5ull,
     0x6a79ad55e7f6fd10ull, 0x6a2ff94f04b962b0ull, 0x69e6784cc2cd61bdull, 0x699d2a2bd181482aull,
     0x69540ec8f895722dull, 0x690b2601182b5e56ull, 0x68c26fb128b4cd63ull, 0x6879ebb63ae2edc6ull,
     0x683199ed779592caull, 0x67e97a341fca775bull, 0x67a18c678c8c8c61ull, 0x6759d0652ee352afull,
     0x6712460a8fc24072ull, 0x66caed354ff83222ull, 0x6683c5c3281ee6e9ull, 0x663ccf91e88a8873ull,
     0x65f60a7f79393e2eull, 0x65af7669d9c2cbe4ull, 0x6569132f21483ba7ull, 0x6522e0ad7e639312ull,
     0x64dcdec3371793d1ull, 0x64970d4ea8bf8766ull, 0x64516c2e47ff1623ull, 0x640bfb40a0b22959ull,
     0x63c6ba6455dcd8aeull, 0x6381a978219b628full, 0x633cc85ad5122fbdull, 0x62f816eb585de1edull,
     0x62b39508aa836d6full, 0x626f4291e1603dd5ull, 0x622b1f66299a6599ull, 0x61e72b64c690d8afull,
     0x61a3666d124bb204ull, 0x615fd05e7d6c83e4ull, 0x611c69188f1eb339ull, 0x60d9307ae507dd9aull,
     0x6096266533384a2bull, 0x60534ab7441b6546ull, 0x60109d50f86846d8ull, 0x5fce1e124712437cull,
     0x5f8bccdb3d398841ull, 0x5f49a98bfe1bc11cull, 0x5f07b404c304c9f1ull, 0x5ec5ec25db3f6a41ull,
     0x5e8451cfac061b5full, 0x5e42e4e2b073d935ull, 0x5e01a53f7974fd86ull, 0x5dc092c6adb825b8ull,
     0x5d7fad59099f22feull, 0x5d3ef4d75f2ff504ull, 0x5cfe69229605cef5ull, 0x5cbe0a1bab4226dfull,
     0x5c7dd7a3b17dcf75ull, 0x5c3dd19bd0ba1c1aull, 0x5bfdf7e546520f3eull, 0x5bbe4a6164eb92f4ull,
     0x5b7ec8f19468bbc9ull, 0x5b3f737751d915c8ull, 0x5b0049d42f6afbb6ull, 0x5ac14be9d45cf869ull,
     0x5a827999fcef3242ull, 0x5a43d2c67a54e0c0ull, 0x5a05575132a5cc20ull, 0x59c7071c20cfd70cull,
     0x5988e20954889245ull, 0x594ae7faf23eda52ull, 0x590d18d3330c7f1eull, 0x58cf747464a7f584ull,
     0x5891fac0e95612c8ull, 0x5854ab9b37dbd1e5ull, 0x581786e5db7022c2ull, 0x57da8c8373adc331ull,
     0x579dbc56b48521baull, 0x57611642662e4a33ull, 0x57249a29651adc07ull, 0x56e847eea1e80a49ull,
     0x56ac1f752150a563ull, 0x5670209ffc1f2e82ull, 0x56344b525f1ff495ull, 0x55f89f6f8b133af4ull,
     0x55bd1cdad49f699cull, 0x5581c377a44346f0ull, 0x5546932976483b15ull, 0x550b8bd3dab49cbdull,
     0x54d0ad5a753e077cull, 0x5495f7a0fd3bbb8eull, 0x545b6a8b3d990704ull, 0x542105fd14c7b869ull,
     0x53e6c9da74b29ab5ull, 0x53acb60762affaaeull, 0x5372ca67f774358full, 0x533906e05f045106ull,
     0x52ff6b54d8a89c75ull, 0x52c5f7a9b6df5b77ull, 0x528cabc35f4f799dull, 0x525387864abb4762ull,
     0x521a8ad704f3404full, 0x51e1b59a2cc8da3eull, 0x51a907b474015dc9ull, 0x5170810a9f48c7cfull,
     0x513821818624b40cull, 0x50ffe8fe12e750c4ull, 0x50c7d76542a25b72ull, 0x508fec9c251a267cull,
     0x50582887dcb8a7e1ull, 0x50208b0d9e8090dfull, 0x4fe91412b2006e83ull, 0x4fb1c37c7145d328ull,
     0x4f7a993048d088d7ull, 0x4f439513b785cc80ull, 0x4f0cb70c4ea39210ull, 0x4ed5feffb1b3d155ull,
     0x4e9f6cd3967fdba8ull, 0x4e69006dc503ba65ull, 0x4e32b9b417619617ull, 0x4dfc988c79d52661ull,
     0x4dc69cdceaa72a9cull, 0x4d90c68b7a20eb1eull, 0x4d5b157e4a7fc325ull, 0x4d25899b8fe8b365ull,
     0x4cf022c9905bfd32ull, 0x4cbae0eea3a8c63cull, 0x4c85c3f13360c4d5ull, 0x4c50cbb7bacbf4cbull,
     0x4c1bf828c6dc54b8ull, 0x4be7492af621abd6ull, 0x4bb2bea4f8bd5847ull, 0x4b7e587d905625d1ull,
     0x4b4a169b900c2d00ull, 0x4b15f8e5dc6cbab0ull, 0x4ae1ff436b663ff7ull, 0x4aae299b443c4a6bull,
     0x4a7a77d47f7b84b1ull, 0x4a46e9d646edbf6aull, 0x4a137f87d58e025bull, 0x49e038d0777ca5e0ull,
     0x49ad159789f37496ull, 0x497a15c47b39d53eull, 0x4947393eca98fcd6ull, 0x49147fee085028d6ull,
     0x48e1e9b9d588e19bull, 0x48af7689e44b44eaull, 0x487d2645f7725895ull, 0x484af8d5e2a06536ull,
     0x4818ee218a3358eeull, 0x47e70610e3393241ull, 0x47b5408bf36472e2ull, 0x47839d7ad1009a90ull,
     0x47521cc5a2e6a9e0ull, 0x4720be54a071ad01ull, 0x46ef821011734e6bull, 0x46be67e04e28717cull,
     0x468d6fadbf2dd4f3ull, 0x465c9960dd74bd4bull, 0x462be4e23237a6efull, 0x45fb521a56ef0042ull,
     0x45cae0f1f545eb73ull, 0x459a9151c70f0819ull, 0x456a632296394492ull, 0x453a564d3cc4b723ull,
     0x450a6abaa4b77ecdull, 0x44daa053c812abd2ull, 0x44aaf701b0c72feeull, 0x447b6ead78aad636ull,
     0x444c0740496d4294ull, 0x441cc0a35c8cf8eaull, 0x43ed9abffb4c6bc9ull, 0x43be957f7ea712b6ull,
     0x438fb0cb4f468808ull, 0x4360ec8ce577ae44ull, 0x433248adc91fdd02ull, 0x4303c51791b21550ull,
     0x42d561b3e6243d8aull, 0x42a71e6c7ce464afull, 0x4278fb2b1bce0d15ull, 0x424af7d9981f7e98ull,
     0x421d1461d66f2023ull, 0x41ef50adcaa0d899ull, 0x41c1aca777db771bull, 0x41942838f07e22a3ull,
     0x4166c34c5615d0ecull, 0x41397dcbd952c4a6ull, 0x410c57a1b9fe12f6ull, 0x40df50b846ef302bull,
     0x40b268f9de0183baull, 0x4085a050ec0a036aull, 0x4058f6a7ecccd5b6ull, 0x402c6be96af2fb58ull},
    {0x8000000000000000ull, 0x7fffa74712c3cdfdull, 0x7fff4e8e6306ed59ull, 0x7ffef5d5f0c93372ull,
     0x7ffe9d1dbc0a75aaull, 0x7ffe4465c4ca895full, 0x7ffdebae0b0943f2ull, 0x7ffd92f68ec67ac3ull,
     0x7ffd3a3f50020332ull, 0x7ffce1884ebbb29full, 0x7ffc88d18af35e6bull, 0x7ffc301b04a8dbf6ull,
     0x7ffbd764bbdc00a2ull, 0x7ffb7eaeb08ca1cdull, 0x7ffb25f8e2ba94dbull, 0x7ffacd435265af2bull,
     0x7ffa748dff8dc61full, 0x7ffa1bd8ea32af18ull, 0x7ff9c32412543f77ull, 0x7ff96a6f77f24c9eull,
     0x7ff911bb1b0cabeeull, 0x7ff8b906fba332c9ull, 0x7ff8605319b5b692ull, 0x7ff8079f75440ca9ull,
     0x7ff7aeec0e4e0a71ull, 0x7ff75638e4d3854cull, 0x7ff6fd85f8d4529cull, 0x7ff6a4d34a5047c4ull,
     0x7ff64c20d9473a26ull, 0x7ff5f36ea5b8ff25ull, 0x7ff59abcafa56c24ull, 0x7ff5420af70c5685ull,
     0x7ff4e9597bed93abull, 0x7ff490a83e48f8faull, 0x7ff437f73e1e5bd4ull, 0x7ff3df467b6d919eull,
     0x7ff38695f6366fb9ull, 0x7ff32de5ae78cb8bull, 0x7ff2d535a4347a77ull, 0x7ff27c85d76951dfull,
     0x7ff223d648172729ull, 0x7ff1cb26f63dcfb9ull, 0x7ff17277e1dd20f2ull, 0x7ff119c90af4f038ull,
     0x7ff0c11a718512f0ull, 0x7ff0686c158d5e7full, 0x7ff00fbdf70da849ull, 0x7fefb7101605c5b3ull,
     0x7fef5e6272758c21ull, 0x7fef05b50c5cd0f8ull, 0x7feead07e3bb699full, 0x7fee545af8912b78ull,
     0x7fedfbae4addebebull, 0x7feda301daa1805cull, 0x7fed4a55a7dbbe31ull, 0x7fecf1a9b28c7ad0ull,
     0x7fec98fdfab38b9eull, 0x7fec40528050c601ull, 0x7febe7a74363ff5eull, 0x7feb8efc43ed0d1dull,
     0x7feb365181ebc4a4ull, 0x7feadda6fd5ffb58ull, 0x7fea84fcb649869full, 0x7fea2c52aca83be2ull,
     0x7fe9d3a8e07bf086ull, 0x7fe97aff51c479f2ull, 0x7fe922560081ad8dull, 0x7fe8c9acecb360bdull,
     0x7fe87104165968ebull, 0x7fe8185b7d739b7dull, 0x7fe7bfb32201cddbull, 0x7fe7670b0403d56cull,
     0x7fe70e6323798797ull, 0x7fe6b5bb8062b9c5ull, 0x7fe65d141abf415dull, 0x7fe6046cf28ef3c8ull,
     0x7fe5abc607d1a66cull, 0x7fe5531f5a872eb3ull, 0x7fe4fa78eaaf6204ull, 0x7fe4a1d2b84a15c8ull,
     0x7fe4492cc3571f68ull, 0x7fe3f0870bd6544cull, 0x7fe397e191c789ddull, 0x7fe33f3c552a9584ull,
     0x7fe2e69755ff4ca9ull, 0x7fe28df2944584b6ull, 0x7fe2354e0ffd1314ull, 0x7fe1dca9c925cd2cull,
     0x7fe18405bfbf8868ull, 0x7fe12b61f3ca1a31ull, 0x7fe0d2be654557f1ull, 0x7fe07a1b14311711ull,
     0x7fe02178008d2cfdull, 0x7fdfc8d52a596f1cull, 0x7fdf70329195b2dbull, 0x7fdf17903641cda2ull,
     0x7fdebeee185d94ddull, 0x7fde664c37e8ddf5ull, 0x7fde0daa94e37e56ull, 0x7fddb5092f4d4b69ull,
     0x7fdd5c6807261a9bull, 0x7fdd03c71c6dc155ull, 0x7fdcab266f241503ull, 0x7fdc5285ff48eb0full,
     0x7fdbf9e5ccdc18e7ull, 0x7fdba145d7dd73f3ull, 0x7fdb48a6204cd1a1ull, 0x7fdaf006a62a075bull,
     0x7fda97676974ea8eull, 0x7fda3ec86a2d50a6ull, 0x7fd9e629a8530f0dull, 0x7fd98d8b23e5fb31ull,
     0x7fd934ecdce5ea7dull, 0x7fd8dc4ed352b25eull, 0x7fd883b1072c2841ull, 0x7fd82b1378722191ull,
     0x7fd7d276272473bcull, 0x7fd779d91342f42eull, 0x7fd7213c3ccd7854ull, 0x7fd6c89fa3c3d59bull,
     0x7fd670034825e171ull, 0x7fd6176729f37142ull, 0x7fd5becb492c5a7bull, 0x7fd5662fa5d0728bull,
     0x7fd50d943fdf8edfull, 0x7fd4b4f9175984e5ull, 0x7fd45c5e2c3e2a09ull, 0x7fd403c37e8d53bbull,
     0x7fd3ab290e46d769ull, 0x7fd3528edb6a8a80ull, 0x7fd2f9f4e5f8426eull, 0x7fd2a15b2defd4a3ull,
     0x7fd248c1b351168cull, 0x7fd1f028761bdd99ull, 0x7fd1978f764fff38ull, 0x7fd13ef6b3ed50d7ull,
     0x7fd0e65e2ef3a7e6ull, 0x7fd08dc5e762d9d4ull, 0x7fd0352ddd3abc10ull, 0x7fcfdc96107b240aull,
     0x7fcf83fe8123e730ull, 0x7fcf2b672f34daf3ull, 0x7fced2d01aadd4c1ull, 0x7fce7a39438eaa0bull,
     0x7fce21a2a9d73041ull, 0x7fcdc90c4d873cd3ull, 0x7fcd70762e9ea530ull, 0x7fcd17e04d1d3ec9ull,
     0x7fccbf4aa902df0eull, 0x7fcc66b5424f5b71ull, 0x7fcc0e2019028960ull, 0x7fcbb58b2d1c3e4eull,
     0x7fcb5cf67e9c4faaull, 0x7fcb04620d8292e6ull, 0x7fcaabcdd9cedd73ull, 0x7fca5339e38104c2ull,
     0x7fc9faa62a98de44ull, 0x7fc9a212af163f6bull, 0x7fc9497f70f8fda7ull, 0x7fc8f0ec7040ee6cull,
     0x7fc89859acede72aull, 0x7fc83fc726ffbd53ull, 0x7fc7e734de764659ull, 0x7fc78ea2d35157afull,
     0x7fc736110590c6c6ull, 0x7fc6dd7f75346910ull, 0x7fc684ee223c1401ull, 0x7fc62c5d0ca79d0bull,
     0x7fc5d3cc3476d9a0ull, 0x7fc57b3b99a99f34ull, 0x7fc522ab3c3fc338ull, 0x7fc4ca1b1c391b20ull,
     0x7fc4718b39957c5full, 0x7fc418fb9454bc69ull, 0x7fc3c06c2c76b0b1ull, 0x7fc367dd01fb2ea9ull,
     0x7fc30f4e14e20bc6ull, 0x7fc2b6bf652b1d7cull, 0x7fc25e30f2d6393eull, 0x7fc205a2bde33480ull,
     0x7fc1ad14c651e4b6ull, 0x7fc154870c221f54ull, 0x7fc0fbf98f53b9cfull, 0x7fc0a36c4fe6899bull,
     0x7fc04adf4dda642cull, 0x7fbff252892f1ef8ull, 0x7fbf99c601e48f72ull, 0x7fbf4139b7fa8b0full,
     0x7fbee8adab70e746ull, 0x7fbe9021dc477989ull, 0x7fbe37964a7e1750ull, 0x7fbddf0af614960eull,
     0x7fbd867fdf0acb3bull, 0x7fbd2df505608c4aull, 0x7fbcd56a6915aeb2ull, 0x7fbc7ce00a2a07e8ull,
     0x7fbc2455e89d6d62ull, 0x7fbbcbcc046fb497ull, 0x7fbb73425da0b2fcull, 0x7fbb1ab8f4303e08ull,
     0x7fbac22fc81e2b31ull, 0x7fba69a6d96a4fedull, 0x7fba111e281481b3ull, 0x7fb9b895b41c95faull,
     0x7fb9600d7d826238ull, 0x7fb907858445bbe5ull, 0x7fb8aefdc8667877ull, 0x7fb8567649e46d65ull,
     0x7fb7fdef08bf7027ull, 0x7fb7a56804f75635ull, 0x7fb74ce13e8bf505ull, 0x7fb6f45ab57d220full,
     0x7fb69bd469cab2cbull, 0x7fb6434e5b747cb1ull, 0x7fb5eac88a7a5539ull, 0x7fb59242f6dc11daull,
     0x7fb539bda099880dull, 0x7fb4e13887b28d4bull, 0x7fb488b3ac26f70bull, 0x7fb4302f0df69ac7ull,
     0x7fb3d7aaad214df6ull, 0x7fb37f2689a6e612ull, 0x7fb326a2a3873893ull, 0x7fb2ce1efac21af3ull,
     0x7fb2759b8f5762aaull, 0x7fb21d186146e532ull, 0x7fb1c49570907805ull, 0x7fb16c12bd33f09aull,
     0x7fb113904731246dull, 0x7fb0bb0e0e87e8f6ull, 0x7fb0628c133813b0ull, 0x7fb00a0a55417a15ull,
     0x7fafb188d4a3f19dull, 0x7faf5907915f4fc5ull, 0x7faf00868b736a05ull, 0x7faea805c2e015d9ull,
     0x7fae4f8537a528baull, 0x7fadf704e9c27823ull, 0x7fad9e84d937d990ull, 0x7fad46050605227aull,
     0x7faced85702a285dull, 0x7fac950617a6c0b4ull, 0x7fac3c86fc7ac0faull, 0x7fabe4081ea5feaaull,
     0x7fab8b897e284f40ull, 0x7fab330b1b018837ull, 0x7faada8cf5317f0aull, 0x7faa820f0cb80937ull,
     0x7faa29916194fc38ull, 0x7fa9d113f3c82d89ull, 0x7fa97896c35172a6ull, 0x7fa92019d030a10dull,
     0x7fa8c79d1a658e38ull, 0x7fa86f20a1f00fa5ull, 0x7fa816a466cffad0ull, 0x7fa7be2869052536ull}};
constexpr unsigned long long kLn2 = 0xb17217f7d1cf79acull;  // round(2^64 ln 2)

constexpr int kGen = 512, kThreads = kGen + 32;
constexpr int kTileA = 128 * 128, kTileB = kDig * 32 * 128;

constexpr float kSmall = 1.f / 128;  // k_atable64_mend
constexpr long long kSmallHi = 1LL << 29;

template <int NP>
constexpr size_t smem_bytes() { return 1024 + (size_t)kDig * kTileA + (size_t)NP * kTileB + 4096 + 256; }

// 2^-t as an integer of 62 fraction bits, t57 = t 2^57 >= 0.
__device__ __forceinline__ unsigned long long pow2neg(long long t57, const unsigned long long *T) {
    const unsigned long long t = (unsigned long long)t57;
    const int n = (int)(t >> 57);
    const unsigned long long r = t & 0x1ffffffffffull;  // 41 bits
    const unsigned long long x = __umul64hi(r << 23, kLn2);                    // x 2^80
    const unsigned long long x2 = __umul64hi(x, x) >> 16;                      // x^2 2^80
    const uint32_t x3 = (uint32_t)(((unsigned long long)(uint32_t)(x >> 32) * (uint32_t)(x2 >> 16)) >> 32);  // x^3 2^80
    const unsigned long long e = x - (x2 >> 1) + __umulhi(x3, 0x2aaaaaabu);    // 2^80 (x - x^2/2 + x^3/6)
    const unsigned long long v = __umul64hi(T[(t >> 49) & 255], T[256 + ((t >> 41) & 255)]);  // 62 fraction bits
    const unsigned long long p = v - (__umul64hi(v, e) >> 16);
    return n == 0 ? p : n < 64 ? (p + (1ull << (n - 1))) >> n : 0ull;
}

// Column exponent of B: |s_j L_jm| < 2^e from the factors' exponents.  Block: one (f, itc).
__global__ __launch_bounds__(256) void k_wexp(int ntc, int n, int nm, const double *__restrict__ rootS,
                                              const double *__restrict__ L, int *__restrict__ we) {
    after_previous();
    __shared__ int mx[64];
    const int fc = blockIdx.x, itc = fc % ntc;
    if (threadIdx.x < 64) mx[threadIdx.x] = 0;
    __syncthreads();
    const double *s = rootS + (size_t)fc * n, *l = L + (size_t)itc * n * nm;
    const int lanes = 256 / nm, m = threadIdx.x % nm, lane = threadIdx.x / nm;
    int e = 0;
    if (lane < lanes)
        for (int j = lane; j < n; j += lanes) e = max(e, expo_pair(expo(s[j]), expo(l[(size_t)j * nm + m])));
    atomicMax(&mx[m], e);
    __syncthreads();
    if ((int)threadIdx.x < nm) we[fc * nm + threadIdx.x] = expo_of_pairs(mx[threadIdx.x]);
}

// B digits [(f, itc) np + piece][digit][bw columns][Kp].
__global__ __launch_bounds__(256) void k_wdigits(int ntc, int n, int nm, int np, int bw, int Kp,
                                                 const double *__restrict__ rootS, const double *__restrict__ L,
                                                 const int *__restrict__ we, __nv_bfloat16 *__restrict__ D) {
    after_previous();
    const int blk = blockIdx.x, fc = blk / np, itc = fc % ntc, col = threadIdx.x & 31;
    const int k0 = blockIdx.y * 128 + (threadIdx.x >> 5) * 16, m = (blk - fc * np) * bw + col;
    if (k0 >= Kp || col >= bw) return;
    const bool ok = m < nm;
    const int e = ok ? we[fc * nm + m] : kNone;
    const bool some = e != kNone && e != kBad;
    double v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i)
        v[i] = (some && k0 + i < n) ? rootS[(size_t)fc * n + k0 + i] * L[((size_t)itc * n + k0 + i) * nm + m] : 0.0;
    put_digits<16>(v, some ? e : 0, D + ((size_t)blk * kDig * bw + col) * Kp + k0, (size_t)bw * Kp);
}

template <int NP>
__global__ void __launch_bounds__(kThreads, 1)
    k_atable64_tc(const __grid_constant__ CUtensorMap tmB, int ntc, int n, int nm, int bw, int MT, int nk, int ks_last,
                  const double *__restrict__ f, const double *__restrict__ logc, const double *__restrict__ rootS,
                  const int *__restrict__ we, const int *__restrict__ bad, double *__restrict__ A, uint8_t *__restrict__ small,
                  int *err, int test_skip1) {
    after_previous();
    if (*bad) return;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *sa = smem, *sb = smem + (size_t)kDig * kTileA;
    unsigned long long *T = (unsigned long long *)(sb + (size_t)NP * kTileB);
    uint64_t *bars = (uint64_t *)(T + 512);
    uint64_t *afull = bars, *aempty = bars + 2, *bfull = bars + 4, *done = bars + 5, *tempty = bars + 6;
    uint32_t *tmem_slot = (uint32_t *)(bars + 7);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int mt = blockIdx.x % MT, fc = blockIdx.x / MT, itc = fc % ntc;
    if (tid < kGen) T[tid] = kPow2[tid >> 8][tid & 255];
    if (tid == 0) {
        for (int h = 0; h < 2; ++h) {
            mbar_init(&afull[h], kGen);
            mbar_init(&aempty[h], 1);
        }
        mbar_init(bfull, 1);
        mbar_init(done, 1);
        mbar_init(tempty, kGen);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 16) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(tmem_slot)), "r"(256 * NP)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;
    constexpr int kPassK = kPassMax / kBK;  // K blocks of one exact pass

    if (warp == 16) {
        // ---------------- B loads and MMAs ----------------
        if (lane == 0) {
            bool ok = true;
            for (int kb = 0; kb < nk && ok; ++kb) {
                // the MMAs that read the last B tile are done once both A halves are free
                if (kb > 0) ok = mbar_wait(&aempty[1], (uint32_t)(kb - 1) & 1u, err, 22) &&
                                 mbar_wait(&aempty[0], (uint32_t)(kb - 1) & 1u, err, 22);
                if (!ok) break;
                mbar_expect_tx(bfull, (uint32_t)(NP * kDig * bw * 128));
                for (int p = 0; p < NP; ++p)
                    for (int t = 0; t < kDig; ++t)
                        tma_2d(sb + p * kTileB + t * 32 * 128, &tmB, bfull, kb * kBK, ((fc * NP + p) * kDig + t) * bw);
                const int pass = kb / kPassK;
                if (kb % kPassK == 0 && pass > 0) ok = mbar_wait(tempty, (uint32_t)(pass - 1) & 1u, err, 23);
                ok = mbar_wait(bfull, (uint32_t)kb & 1u, err, 24) && ok;
                const int nks = kb == nk - 1 ? ks_last : kBK / 16;
                for (int h = 0; h < 2 && ok; ++h) {
                    if (!mbar_wait(&afull[h], (uint32_t)kb & 1u, err, 25)) { ok = false; break; }
                    fence_after();
#pragma unroll
                    for (int s = 0; s < kDig; ++s) {
                        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)((kDig - s) * 32 >> 3) << 17) |
                                               ((uint32_t)(128 >> 4) << 24);
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            const int ks = 2 * h + q;
                            if (ks < nks)
                                for (int p = 0; p < NP; ++p)
                                    mma_n(tmem + p * 256 + s * 32, sdesc(su32(sa + s * kTileA) + ks * 32),
                                          sdesc(su32(sb + p * kTileB) + ks * 32), idesc,
                                          (kb % kPassK > 0 || ks > 0 || s > 0) ? 1u : 0u);
                        }
                    }
                    mma_commit(&aempty[h]);
                }
                if (ok && (kb % kPassK == kPassK - 1 || kb == nk - 1) && !(test_skip1 == pass + 1 && blockIdx.x == 0))
                    mma_commit(done);
            }
            if (!ok) {  // what is in flight lands before the block leaves
                mma_commit(done);
                const uint64_t t0 = gtime();
                while (gtime() - t0 < kWaitNs / 100) {
                }
            }
        }
        __syncwarp();
    } else {
        // ---------------- digits of c_ij^|f|, then the sums ----------------
        const int row = 8 * warp + ((lane >> 3) & 3) + 4 * ((lane >> 2) & 1), gi = mt * 128 + row;
        const double af = fabs(f[fc / ntc]);
        // t57 = log c x (-|f| log2(e) 2^57)
        const double k57 = -af * 1.4426950408889634073599246810019 * 144115188075855872.0;
        const double *lc = logc + ((size_t)itc * n + min(gi, n - 1)) * n;
        const int quarter = warp & 3, cg = warp >> 2;  // TMEM lanes and columns of this warp
        long long hi[NP][8], lo[NP][8];
#pragma unroll
        for (int p = 0; p < NP; ++p)
#pragma unroll
            for (int q = 0; q < 8; ++q) hi[p][q] = lo[p][q] = 0;
        bool ok = true;
        for (int kb = 0; kb < nk && ok; ++kb) {
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
                const int chunk = 4 * h + (lane & 3), j0 = kb * kBK + chunk * 8;
                double l[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) l[q] = j0 + q < n ? lc[j0 + q] : 0.0;
                if (kb > 0 && !mbar_wait(&aempty[h], (uint32_t)(kb - 1) & 1u, err, 21)) ok = false;
                if (gi < n) {  // rows past the matrix are never read back
                    uint32_t w[kDig][4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        uint32_t d[2][kDig];
#pragma unroll
                        for (int z = 0; z < 2; ++z) {
                            const int j = j0 + 2 * q + z;
                            const unsigned long long x = j >= n       ? 0ull
                                                         : af == 0.0 ? 1ull << 62
                                                                     : pow2neg(__double2ll_rn(l[2 * q + z] * k57), T);
                            digits_of(x, d[z]);
                        }
#pragma unroll
                        for (int s = 0; s < kDig; ++s) w[s][q] = __byte_perm(d[0][s], d[1][s], 0x7632);
                    }
                    const uint32_t o = (uint32_t)(row * 128 + ((chunk ^ (row & 7)) << 4));
#pragma unroll
                    for (int s = 0; s < kDig; ++s)
                        *reinterpret_cast<uint4 *>(sa + s * kTileA + o) = make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                mbar_arrive(&afull[h]);
            }
            // where a wait failed the lanes may differ: leave together, the warp-wide steps below need them all
            ok = __all_sync(0xffffffffu, ok);
            if (kb % kPassK == kPassK - 1 || kb == nk - 1) {
                const uint32_t ph = (uint32_t)(kb / kPassK) & 1u;
                ok = __all_sync(0xffffffffu, mbar_wait(done, ph, err, 26)) && ok;
                fence_after();
                if (ok) {
#pragma unroll
                    for (int p = 0; p < NP; ++p) {
#pragma unroll
                        for (int z = 0; z < 2; ++z) {
                            uint32_t v[4][8];
#pragma unroll
                            for (int t = 0; t < 4; ++t)
                                tmem_ld8(tmem + ((uint32_t)(quarter * 32) << 16) + p * 256 + (4 * z + t) * 32 + cg * 8, v[t]);
                            tmem_wait_ld();
#pragma unroll
                            for (int q = 0; q < 8; ++q) {
                                int D[4];
#pragma unroll
                                for (int t = 0; t < 4; ++t) D[t] = __float2int_rn(__uint_as_float(v[t][q]));
                                (z ? lo : hi)[p][q] += join_levels(D);
                            }
                        }
                    }
                }
                fence_before();
                mbar_arrive(tempty);
            }
        }
        const int r = quarter * 32 + lane, ri = mt * 128 + r;
        if (ok && ri < n) {
            const double si = rootS[(size_t)fc * n + ri];
            double *out = A + ((size_t)fc * n + ri) * nm;
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                if (cg * 8 >= bw) continue;
                uint32_t mask = 0;  // bit q: the sum is below kSmall of its scale, k_atable64_mend looks
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int m = p * bw + cg * 8 + q;
                    if (m >= nm) continue;
                    const int e = we[fc * nm + m];
                    const long long h = hi[p][q] + (lo[p][q] >> 32);
                    if (e == kBad || (e != kNone && h < kSmallHi && h >= -kSmallHi)) mask |= 1u << q;
                    out[m] = e == kBad || e == kNone ? 0.0 : si * combine(hi[p][q], lo[p][q], e - 68);
                }
                small[((size_t)fc * n + ri) * 8 + p * (bw / 8) + cg] = (uint8_t)mask;
            }
        }
    }
    fence_before();
    __syncthreads();
    fence_after();
    if (warp == 16) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256 * NP) : "memory");
}

// Rows where c_ij^|f| decays between i and the nodes that a mode moves: the digits' error is absolute
// against the largest s_j L_jm (2^-62 a term), so an element keeps them only where sum_j c_ij^|f| |s_j
// L_jm| >= kSmall of the scale.  Measured error relative to that sum from the line to twice it, digits / FP64
// pipe: 200 nodes 1.2e-16 / 2.8e-16, 400 1.4e-16 / 3.7e-16, 1000 with local modes 3.7e-16 / 8.3e-16, 1200 1.4e-16
// / 2.7e-16; below half of it the digits' is the larger.  The element itself and then the 32 nodes around i
// bound the sum from below; what is left is summed on the FP64 pipe, lanes over j, without the nodes that add
// less than 2^-60 of it (zones of 200 nodes 85 -> 35 us, 400 nodes x 2 100 -> 44).
// A warp scans the masks of eight rows, far apart (those near the foot of a tower come together: 32
// neighbouring rows a warp took twice the time).
__global__ __launch_bounds__(256) void k_atable64_mend(int rows, int ntc, int n, int nm, const double *__restrict__ f,
                                                       const double *__restrict__ logc, const double *__restrict__ expt,
                                                       const double *__restrict__ rootS, const double *__restrict__ L,
                                                       const int *__restrict__ we, const int *__restrict__ bad,
                                                       const unsigned long long *__restrict__ small, double *__restrict__ A) {
    after_previous();
    if (*bad) return;
    __shared__ double T[kExpTab];
    T[threadIdx.x] = expt[threadIdx.x];
    __syncthreads();
    const int lane = threadIdx.x & 31, first = blockIdx.x * 8 + (threadIdx.x >> 5), step = gridDim.x * 8;
    const unsigned long long own = lane < 8 && first + lane * step < rows ? small[first + lane * step] & (~0ull >> (64 - nm)) : 0ull;
    for (unsigned todo = __ballot_sync(0xffffffffu, own != 0); todo; todo &= todo - 1) {
        const int src = __ffs(todo) - 1, row = first + src * step, fc = row / n, i = row - fc * n, itc = fc % ntc;
        unsigned long long mk = __shfl_sync(0xffffffffu, own, src);
        const double af = fabs(f[fc / ntc]);
        const double *lc = logc + ((size_t)itc * n + i) * n, *s = rootS + (size_t)fc * n, *l = L + (size_t)itc * n * nm;
        const int jw = max(0, min(i - 16, n - 32)) + lane;
        const float cw = jw >= n ? 0.f : af == 0.0 ? 1.f : expf((float)(af * lc[jw]));
        float least = 1.f;  // of the sums that are too small, over the 32 nodes
        for (unsigned long long b = mk; b; b &= b - 1) {
            const int m = __ffsll(b) - 1, e = we[fc * nm + m];
            if (e == kBad) {  // the whole column
                least = 0.f;
                continue;
            }
            float v = jw < n ? cw * scaled_abs(s[jw] * l[(size_t)jw * nm + m], e) : 0.f;
#pragma unroll
            for (int h = 16; h > 0; h >>= 1) v += __shfl_xor_sync(0xffffffffu, v, h);
            if (v >= kSmall) mk &= ~(1ull << m);
            else least = fminf(least, v);
        }
        // nodes that add less than 2^-60 of every sum are passed over, 32 at a time (scaled_abs is true to 2^-60)
        const float skip = least >= 0x1p-40f ? least * 0x1p-60f / (float)n : -1.f;
        while (mk) {
            int m[8], cnt = 0;
            double acc[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                m[q] = 0;
                acc[q] = 0.0;
                if (mk) {
                    m[q] = __ffsll(mk) - 1;
                    mk &= mk - 1;
                    ++cnt;
                }
            }
            for (int j0 = 0; j0 < n; j0 += 32) {
                const int j = j0 + lane;
                const bool in = j < n;
                const double x = in ? af * lc[j] : 0.0;
                if (!__any_sync(0xffffffffu, in && (af == 0.0 || expf((float)x) > skip))) continue;
                const double c = !in ? 0.0 : af == 0.0 ? 1.0 : expc(x, T), sj = in ? s[j] : 0.0;
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    if (in && q < cnt) acc[q] = fma(c, sj * l[(size_t)j * nm + m[q]], acc[q]);
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                if (q >= cnt) continue;
                for (int h = 16; h > 0; h >>= 1) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], h);
                if (lane == 0) A[(size_t)row * nm + m[q]] = s[i] * acc[q];
            }
        }
    }
}

template <int NP>
static cudaError_t launch(cudaStream_t st, const CUtensorMap &mb, int nf, const double *f, int ntc, int n, int nm, int bw,
                          const double *logc, const double *rootS, const int *we, const int *bad, double *A, uint8_t *small,
                          int *err, int test_skip1) {
    const int MT = (n + 127) / 128, nk = (n + kBK - 1) / kBK, ks_last = (n - (nk - 1) * kBK + 15) / 16;
    cudaError_t e = cudaFuncSetAttribute(k_atable64_tc<NP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<NP>());
    if (e != cudaSuccess) return e;
    launch_next(k_atable64_tc<NP>, (unsigned)(nf * ntc * MT), kThreads, smem_bytes<NP>(), st, mb, ntc, n, nm, bw, MT, nk, ks_last, f, logc,
                                                                                   rootS, we, bad, A, small, err, test_skip1);
    return cudaGetLastError();
}

}  // namespace at64

// [digits][exponents][masks, 8 bytes a row] of nf frequencies
static size_t up256(size_t n) { return (n + 255) & ~(size_t)255; }
size_t atable64_tc_scratch(int nf, int ntc, int nnl, int nm) {
    const size_t nb = (size_t)nf * ntc * p64::blocks_of(nm), Kp = (nnl + tc::kBK - 1) / tc::kBK * tc::kBK;
    return up256(nb * p64::kDig * p64::block_width(nm) * Kp * 2) + up256(sizeof(int) * (size_t)nf * ntc * nm) +
           (size_t)8 * nf * ntc * nnl;
}

cudaError_t launch_atable64_tc(cudaStream_t st, int nf, const double *f, int ntc, int nnl, int nm, const double *logc,
                               const double *rootS, const double *L, const int *bad, double *A, void *scratch, int *err,
                               int test_skip1) {
    using namespace at64;
    const int np = blocks_of(nm), bw = block_width(nm), Kp = (nnl + kBK - 1) / kBK * kBK, rows = nf * ntc * nnl;
    const size_t nb = (size_t)nf * ntc * np;
    __nv_bfloat16 *D = (__nv_bfloat16 *)scratch;
    int *we = (int *)((char *)scratch + up256(nb * kDig * bw * Kp * 2));
    uint8_t *small = (uint8_t *)we + up256(sizeof(int) * (size_t)nf * ntc * nm);
    launch_next(k_wexp, nf * ntc, 256, 0, st, ntc, nnl, nm, rootS, L, we);
    launch_next(k_wdigits, dim3((unsigned)nb, (Kp + 127) / 128), 256, 0, st, ntc, nnl, nm, np, bw, Kp, rootS, L, we, D);
    CUtensorMap mb;
    if (!make_map(&mb, D, Kp, (uint64_t)nb * kDig * bw, (uint32_t)bw)) return cudaErrorInvalidValue;
    const cudaError_t e = np == 1 ? launch<1>(st, mb, nf, f, ntc, nnl, nm, bw, logc, rootS, we, bad, A, small, err, test_skip1)
                                  : launch<2>(st, mb, nf, f, ntc, nnl, nm, bw, logc, rootS, we, bad, A, small, err, test_skip1);
    if (e != cudaSuccess) return e;
    launch_next(k_atable64_mend, (unsigned)((rows + 63) / 64), 256, 0, st, rows, ntc, nnl, nm, f, logc,
                logc + (size_t)ntc * nnl * nnl, rootS, L, we, bad, (const unsigned long long *)small, A);
    return cudaGetLastError();
}

}  // namespace bsa
